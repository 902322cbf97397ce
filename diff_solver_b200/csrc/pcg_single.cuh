// Jacobi-PCG with one grid synchronisation per iteration (included by
// pressure.cu).
//
// The textbook iteration needs two grid-wide sums: p.q before alpha, r.z
// before beta.  Here one pass computes, from alpha and beta of the previous
// one, z_k = z - alpha q, p_k = z_k + beta p and q_k = M^-1 A p_k for a cell
// and, because the operator reads p_k at the six neighbours, z_k and p_k
// again at those (three loads and two fused multiply-adds each).  The pass
// sums
//     r.z, r.r, p.A p, A p.z, A p.M^-1 A p, r.A p, A p.A p
// from which alpha_k and, one step ahead, r_{k+1}.z_{k+1} and r_{k+1}.r_{k+1}
// follow (all in FP64).  r.z and r.r are summed anew from the stored z_k each
// time: the prediction spans one step, in which the residual falls by a small
// factor, so nothing cancels and nothing drifts.  32 bytes per cell and
// iteration (read z, q, p, e; write z, q, p, e) against 36 with two passes.
//
// What bounds it: on grids the SMs can hold, latency -- a 64^3 iteration is
// 4.0 us, 2.6 of them the reduction over 139 blocks (the two-pass kernel: 13.5,
// two reductions of 4.4 to 8.6 and L2 trips for every vector); on larger ones,
// the loads and the instructions of the operator.  Iteration counts are those
// of the two-pass kernel.
#pragma once

namespace xs {

constexpr int kCgThreads = 512;
constexpr int kCgWarps = kCgThreads / 32;
constexpr size_t kCgMaxSmem = 216 * 1024;  // dynamic shared memory a block may ask for
constexpr uint32_t kCodeReal = 0x40u, kCodeGhost = 0x80u, kCodeDiag = 7u;
constexpr uint32_t kCodeReal4 = 0x40404040u;   // the four bytes' real-cell bits
constexpr uint32_t kCodeInner4 = 0x46464646u;  // four cells with all six neighbours, none copied

// The marching form's vectors are padded so that no load needs a boundary
// test: rows of `pitch` floats (a multiple of 4, at least one slot past the
// row), `rows` rows per plane (at least one past the plane) and a plane before
// and after.  A row's x = -1 is the slot before it, which is the last slot of
// the row before.  The padding holds zeros, which is what Neumann and fixed
// faces contribute, and so do solid cells; on periodic axes it holds copies
// that the cell's owner writes with the cell.  A code byte per cell holds the
// diagonal (0: not an unknown), so colliders and ragged extents take the same
// 16-byte loads as everything else.
struct PadGeom {
    uint32_t nx, ny, nz, n;
    uint32_t pitch, rows, plane, base;
    uint32_t total;  // floats per vector
    FastDiv dnx, dny, dpitch, drows;
    uint32_t periodic;  // bit d: axis d wraps

    __device__ __forceinline__ uint32_t at(int x, int y, int z) const {
        return base + static_cast<uint32_t>(x) + pitch * static_cast<uint32_t>(y) + plane * static_cast<uint32_t>(z);
    }
};

// ------------------------------------------------------------- reduction
// Grid-wide sums of K doubles without a serial step: every block publishes
// its K sums, each in 16 bytes beside the epoch that makes it valid, and
// every block adds up all of them itself, in block order (deterministic).
// One store and one load cross the L2 per reduction; the counter that a last
// block must notice, sum for and answer costs four such trips.  Two sets of
// slots alternate: a block can only start the reduction after next when all
// have read this one.
constexpr int kMaxSlotStride = 16;
struct SlotSync {
    ulonglong2* slots;  // [2][blocks * kMaxSlotStride]
    SolverState* st;
    unsigned long long epoch;
};

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void publish16(ulonglong2* p, double v, unsigned long long epoch) {
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(__double_as_longlong(v)), "l"(epoch)
                 : "memory");
}
__device__ __forceinline__ void observe16(const ulonglong2* p, unsigned long long& v, unsigned long long& epoch) {
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}" : "=l"(v), "=l"(epoch) : "l"(p) : "memory");
}

constexpr int slot_stride(int k) { return k <= 1 ? 1 : (k <= 2 ? 2 : (k <= 4 ? 4 : (k <= 8 ? 8 : 16))); }

template <int K>
__device__ bool slot_reduce(SlotSync& s, double (&v)[K]) {
    constexpr int KP = slot_stride(K);
    constexpr int kParts = 32 / KP;
    __shared__ double block_part[kCgWarps][KP], grid_part[kCgWarps][KP];
    __shared__ unsigned failed;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // warp sums, halving the number of values with the lanes that hold them
    double w[KP];
#pragma unroll
    for (int k = 0; k < KP; ++k) w[k] = k < K ? v[k] : 0.0;
    int index = 0;
#pragma unroll
    for (int h = KP / 2, m = 16; m >= 1; h /= 2, m /= 2) {
        if (h >= 1) {
            const bool upper = (lane & m) != 0;
            index |= upper ? h : 0;
#pragma unroll
            for (int i = 0; i < h; ++i) {
                const double keep = upper ? w[i + h] : w[i], give = upper ? w[i] : w[i + h];
                w[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
            }
        } else {
            w[0] += __shfl_xor_sync(0xffffffffu, w[0], m);
        }
    }
    if ((lane & (kParts - 1)) == 0) block_part[warp][index] = w[0];
    if (threadIdx.x == 0) failed = 0u;
    __syncthreads();
    const unsigned long long epoch = ++s.epoch;
    ulonglong2* slots = s.slots + static_cast<size_t>(epoch & 1u) * gridDim.x * kMaxSlotStride;  // (apart for every K)
    const int k = lane & (KP - 1), part = lane / KP;
    if (warp == 0) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < (kCgWarps + kParts - 1) / kParts; ++q) {
            const int j = part + q * kParts;
            t += j < kCgWarps ? block_part[j][k] : 0.0;
        }
#pragma unroll
        for (int m = KP; m < 32; m *= 2) t += __shfl_xor_sync(0xffffffffu, t, m);
        fence_gpu();  // the block's writes (ordered by the barrier above) before its sums
        if (lane < KP) publish16(slots + static_cast<size_t>(blockIdx.x) * KP + lane, t, epoch);
    }
    double acc = 0.0;
    const long long t0 = clock64();
    for (uint32_t e = threadIdx.x; e < gridDim.x * KP; e += kCgThreads) {
        unsigned long long bits, seen;
        observe16(slots + e, bits, seen);
        while (seen != epoch) {
            if (clock64() - t0 > kBarrierTimeoutCycles) {
                atomicExch(&s.st->error, 1u);
                failed = 1u;
                break;
            }
            observe16(slots + e, bits, seen);
        }
        acc += __longlong_as_double(static_cast<long long>(bits));
    }
    fence_gpu();  // the other blocks' writes after their sums
#pragma unroll
    for (int m = KP; m < 32; m *= 2) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (lane < KP) grid_part[warp][lane] = acc;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < (kCgWarps + kParts - 1) / kParts; ++q) {
        const int j = part + q * kParts;
        t += j < kCgWarps ? grid_part[j][k] : 0.0;
    }
#pragma unroll
    for (int m = KP; m < 32; m *= 2) t += __shfl_xor_sync(0xffffffffu, t, m);
#pragma unroll
    for (int i = 0; i < K; ++i) v[i] = __shfl_sync(0xffffffffu, t, i);
    return failed == 0u;
}

// ----------------------------------------------------------------- phases
struct BrickGeom {
    uint32_t row_quads;      // 4-cell groups per row, the last one partial when nx is no multiple of 4
    uint32_t by, bz;         // rows of a brick
    uint32_t bricks_y;       // bricks along y
};

struct CgArgs {
    PcgArgs c;  // right-hand side, guess, x64, outputs, tolerance (z .. y unused)
    PadGeom g;
    float* z[2];
    float* p[2];
    float* q[2];
    float* e;
    float* s;
    float* y;
    uint8_t* code;
    ulonglong2* slots;
    // the marching form: runs of `run` groups of a plane, slabs of `slab` planes
    uint32_t run, runs, slab, slabs;
    BrickGeom brick;  // the resident form
};

// Copies of a cell's value for its periodic neighbours.
__device__ __forceinline__ void store_copies(const PadGeom& g, float* v, int x, int y, int z, float value) {
    if (g.periodic & 1u) {
        if (x == 0) v[g.at(static_cast<int>(g.nx), y, z)] = value;
        if (x == static_cast<int>(g.nx) - 1) v[g.at(-1, y, z)] = value;
    }
    if (g.periodic & 2u) {
        if (y == 0) v[g.at(x, static_cast<int>(g.ny), z)] = value;
        if (y == static_cast<int>(g.ny) - 1) v[g.at(x, -1, z)] = value;
    }
    if (g.periodic & 4u) {
        if (z == 0) v[g.at(x, y, static_cast<int>(g.nz))] = value;
        if (z == static_cast<int>(g.nz) - 1) v[g.at(x, y, -1)] = value;
    }
}

// Codes of the real cells, and zeros in the padding.  A slot that holds a
// periodic copy of z gets it from its owner in residual_pad, unordered with
// this pass: it is left alone here.
static __device__ __noinline__ void pad_phase(const CgArgs& a) {
    const PadGeom& g = a.g;
    const Grid& grid = a.c.op.g;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < g.total; j += gridDim.x * blockDim.x) {
        const uint32_t row = fastdiv(j, g.dpitch), zz = fastdiv(row, g.drows);
        int x = static_cast<int>(j - row * g.pitch), y = static_cast<int>(row - zz * g.rows), z = static_cast<int>(zz) - 1;
        if (x < grid.nx && y < grid.ny && z >= 0 && z < grid.nz) {
            CellStencil s;
            const uint64_t i = idx3(x, y, z, grid.nx, grid.ny);
            const bool act = stencil(a.c.op, x, y, z, i, s);
            uint32_t code = kCodeReal | (act ? static_cast<uint32_t>(s.diag) : 0u);
            if (((g.periodic & 1u) && (x == 0 || x == grid.nx - 1)) || ((g.periodic & 2u) && (y == 0 || y == grid.ny - 1)) ||
                ((g.periodic & 4u) && (z == 0 || z == grid.nz - 1)))
                code |= kCodeGhost;
            a.code[j] = static_cast<uint8_t>(code);
            continue;
        }
        a.code[j] = 0;
        // the last slot of a row is x = -1 of the next one, the last row of a plane y = -1 of the next
        int cx = x, cy = y, cz = z;
        if (x == static_cast<int>(g.pitch) - 1) {
            cx = -1;
            if (++cy == static_cast<int>(g.rows)) { cy = 0; ++cz; }
        }
        bool copy = (g.periodic & 1u) && (cx == -1 || cx == grid.nx) && cy < grid.ny && cz >= 0 && cz < grid.nz;
        if ((g.periodic & 2u) && x < grid.nx) {
            const bool low = y == static_cast<int>(g.rows) - 1, high = y == grid.ny;
            copy = copy || (low && z + 1 >= 0 && z + 1 < grid.nz) || (high && z >= 0 && z < grid.nz);
        }
        copy = copy || ((g.periodic & 4u) && x < grid.nx && y < grid.ny && (z == -1 || z == grid.nz));
        if (!copy) a.z[0][j] = 0.0f;
        a.z[1][j] = 0.0f;
        a.p[0][j] = 0.0f;
        a.p[1][j] = 0.0f;
        a.q[0][j] = 0.0f;
        a.q[1][j] = 0.0f;
    }
}

// Where a pass' first residual goes.  Padded vectors: z with its periodic
// copies, p = q = e = 0.
struct PadStore {
    const CgArgs& a;
    __device__ __forceinline__ void quad(int x, int y, int z, const float4& v) const {
        const uint32_t j = a.g.at(x, y, z);
        const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        st4(a.z[0] + j, v);
        st4(a.p[0] + j, zero4);
        st4(a.q[0] + j, zero4);
        st4(a.e + j, zero4);
        if (a.g.periodic) {
            const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) store_copies(a.g, a.z[0], x + k, y, z, f[k]);
        }
    }
    __device__ __forceinline__ void cell(int x, int y, int z, float v) const {
        const uint32_t j = a.g.at(x, y, z);
        a.z[0][j] = v;
        a.p[0][j] = 0.0f;
        a.q[0][j] = 0.0f;
        a.e[j] = 0.0f;
        if (a.g.periodic) store_copies(a.g, a.z[0], x, y, z, v);
    }
};

// r = b - A x in FP64 for the zero start, the scaled guess or the iterate x64
// (as residual_phase); z = r / diag goes to `out`.  v = {b.b, r.r, r.z}.
template <class Store>
__device__ __noinline__ void residual_to(const PcgArgs& c, const Store& out, int mode, double (&v)[3], double scale) {
    const Grid& g = c.op.g;
    v[0] = v[1] = v[2] = 0.0;
    if (c.fast_residual) {
        const FastGeom& f = c.fast;
        for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < f.groups; t += gridDim.x * blockDim.x) {
            const uint32_t i = 4u * t;
            double xi[4] = {0.0, 0.0, 0.0, 0.0}, ax[4] = {0.0, 0.0, 0.0, 0.0};
            float4 d4;
            const uint32_t row = fastdiv(i, f.dnx), z = fastdiv(row, f.dny), y = row - z * f.ny, x = i - row * f.nx;
            if (mode == kFromGuess) {
                apply4_fp64(f, guess_view(c), i, xi, ax, d4);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    xi[k] *= scale;
                    ax[k] *= scale;
                }
            } else if (mode == kFromX64) {
                apply4_fp64(f, c.x64, i, xi, ax, d4);
            } else {
                const RowGeom rg = row_geom(f, y, z);
                int32_t left, right;
                x_geom(f, x, rg.dyz, left, right, d4);
            }
            const float dd[4] = {d4.x, d4.y, d4.z, d4.w};
            float zf[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double b = rhs_at4(c, i, k);
                const double r = b - ax[k];
                zf[k] = static_cast<float>(r / dd[k]);
                v[0] += b * b;
                v[1] += r * r;
                v[2] += r * static_cast<double>(zf[k]);
                if (mode != kFromX64) c.x64[i + k] = xi[k];
                if (c.solution_out) c.solution_out[i + k] = xi[k];
            }
            out.quad(static_cast<int>(x), static_cast<int>(y), static_cast<int>(z), make_float4(zf[0], zf[1], zf[2], zf[3]));
            if (c.pressure_out)
                st4(c.pressure_out + i, make_float4(static_cast<float>(xi[0]), static_cast<float>(xi[1]), static_cast<float>(xi[2]),
                                                    static_cast<float>(xi[3])));
        }
        return;
    }
    const uint64_t n = cell_count(g);
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        int x, y, z;
        decode(i, g.nx, g.ny, x, y, z);
        CellStencil s;
        const bool act = stencil(c.op, x, y, z, i, s);
        const double b = act ? rhs_at(c, i) + static_cast<double>(s.fixed_sum) : 0.0;
        double xi = 0.0, ax = 0.0;
        if (act && mode == kFromGuess) {
            const GuessView guess = guess_view(c);
            xi = guess[i];
            ax = s.diag * xi;
#pragma unroll
            for (int f = 0; f < 6; ++f)
                if ((s.conn >> f) & 1u) { const uint64_t j = s.nb[f]; if (j != c.op.anchor) ax -= guess[j]; }
            xi *= scale;
            ax *= scale;
        } else if (act && mode == kFromX64) {
            xi = c.x64[i];
            ax = s.diag * xi;
#pragma unroll
            for (int f = 0; f < 6; ++f)
                if ((s.conn >> f) & 1u) ax -= c.x64[s.nb[f]];
        }
        if (mode != kFromX64) c.x64[i] = xi;
        const double r = b - ax;
        const float zf = act ? static_cast<float>(r / s.diag) : 0.0f;
        out.cell(x, y, z, zf);
        if (c.pressure_out) c.pressure_out[i] = static_cast<float>(xi);
        if (c.solution_out) c.solution_out[i] = xi;
        v[0] += b * b;
        v[1] += r * r;
        v[2] += r * static_cast<double>(zf);
    }
}

enum CgSum { kRZ = 0, kRR, kPQ, kQZ, kQMQ, kRQ, kQQ, kSR, kSS, kSQ };
template <bool kSmooth>
constexpr int kCgSums = kSmooth ? 10 : 7;

// A vector's value for a group of four cells: one 16-byte store, or cell by
// cell where the group has periodic copies, or ends its row beside slots that
// hold some.
__device__ __forceinline__ bool plain_store(const PadGeom& g, uint32_t c4) {
    return (c4 & (kCodeGhost * 0x01010101u)) == 0u && ((g.periodic & 1u) == 0u || (c4 & kCodeReal4) == kCodeReal4);
}
static __device__ __noinline__ void store_edge(const PadGeom& g, float* v, uint32_t i, uint32_t c4, float4 w) {
    const uint32_t j = i - g.base, row = fastdiv(j, g.dpitch), zz = fastdiv(row, g.drows);
    const int x = static_cast<int>(j - row * g.pitch), y = static_cast<int>(row - zz * g.rows), z = static_cast<int>(zz);
    const float f[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        if (((c4 >> (8 * m)) & kCodeReal) == 0u) continue;
        v[i + m] = f[m];
        store_copies(g, v, x + m, y, z, f[m]);
    }
}
__device__ __forceinline__ void store_quad(const PadGeom& g, float* v, uint32_t i, uint32_t c4, const float4& w) {
    if (plain_store(g, c4)) st4(v + i, w);
    else store_edge(g, v, i, c4, w);
}

// What iteration k reads and writes; alpha, beta: of the step that led to
// z_k.  With smoothing active, s and y advance to step k - 1 by eta
// (s += eta (r_{k-1} - s), y += eta (e_{k-1} - y)) and are summed against
// r_k and A p_k; starting, s = r_k and y = e_k.
struct CgStep {
    // (no __restrict__: other blocks write what a later pass reads)
    const float *zo, *po, *qo;
    float *zw, *pw, *qw;
    float alpha, beta, eta;
    int smooth;
};

struct CgQuad {
    float4 z, p, s;  // z_k, p_k, and the smoothed residual of step k - 1
    uint32_t c4;
};

struct CgLoad {
    float4 z, q, p;
};

__device__ __forceinline__ CgLoad cg_load(const CgStep& k, uint32_t i) { return CgLoad{ld4(k.zo + i), ld4(k.qo + i), ld4(k.po + i)}; }
__device__ __forceinline__ float4 cg_direction(const CgStep& k, const CgLoad& l) {
    return axpy4(axpy4(l.z, -k.alpha, l.q), k.beta, l.p);
}

__device__ __forceinline__ void cg_diagonal(uint32_t c4, float (&d)[4]) {
#pragma unroll
    for (int m = 0; m < 4; ++m) d[m] = static_cast<float>((c4 >> (8 * m)) & kCodeDiag);
}

// z_k, p_k and e_k of a group, and the smoothed sequence, stored.
template <bool kSmooth>
__device__ __forceinline__ void cg_begin(const CgArgs& a, const CgStep& k, uint32_t i, const CgLoad& l, const float4& eo, CgQuad& u) {
    if ((u.c4 & kCodeReal4) == 0u) return;
    const float4 en = axpy4(eo, k.alpha, l.p);
    store_quad(a.g, k.zw, i, u.c4, u.z);
    store_quad(a.g, k.pw, i, u.c4, u.p);
    st4(a.e + i, en);
    if (kSmooth && k.smooth != kSmoothOff) {
        float d[4];
        cg_diagonal(u.c4, d);
        float4 yn = en;
        if (k.smooth == kSmoothStart) {
            u.s = make_float4(u.z.x * d[0], u.z.y * d[1], u.z.z * d[2], u.z.w * d[3]);
        } else {
            const float4 so = ld4(a.s + i), yo = ld4(a.y + i);
            u.s = make_float4(fmaf(k.eta, fmaf(l.z.x, d[0], -so.x), so.x), fmaf(k.eta, fmaf(l.z.y, d[1], -so.y), so.y),
                              fmaf(k.eta, fmaf(l.z.z, d[2], -so.z), so.z), fmaf(k.eta, fmaf(l.z.w, d[3], -so.w), so.w));
            yn = make_float4(fmaf(k.eta, eo.x - yo.x, yo.x), fmaf(k.eta, eo.y - yo.y, yo.y), fmaf(k.eta, eo.z - yo.z, yo.z),
                             fmaf(k.eta, eo.w - yo.w, yo.w));
        }
        st4(a.s + i, u.s);
        st4(a.y + i, yn);
    }
}

// M^-1 A p_k of a group from the sum over its neighbours, and the group's part
// of the sums.  6 p - sum first, then the division: dividing the
// sum instead shifts the operator by the rounding of 1/6, which the smallest
// eigenvalues of a 256^3 grid feel as 0.5 %.
template <bool kSmooth>
__device__ __forceinline__ float4 cg_operator(const float4& sum, const CgQuad& u, int smooth, double (&v)[kCgSums<kSmooth>]) {
    float4 qn;
    const bool inner = (u.c4 & ~(kCodeGhost * 0x01010101u)) == kCodeInner4;
    float d[4] = {6.0f, 6.0f, 6.0f, 6.0f};
    if (inner) {
        constexpr float r6 = 1.0f / 6.0f;
        qn = make_float4(fmaf(6.0f, u.p.x, -sum.x) * r6, fmaf(6.0f, u.p.y, -sum.y) * r6, fmaf(6.0f, u.p.z, -sum.z) * r6, fmaf(6.0f, u.p.w, -sum.w) * r6);
    } else {  // a cell that is no unknown keeps z = p = q = 0
        cg_diagonal(u.c4, d);
        qn = make_float4(d[0] > 0.0f ? fmaf(d[0], u.p.x, -sum.x) / d[0] : 0.0f, d[1] > 0.0f ? fmaf(d[1], u.p.y, -sum.y) / d[1] : 0.0f,
                         d[2] > 0.0f ? fmaf(d[2], u.p.z, -sum.z) / d[2] : 0.0f, d[3] > 0.0f ? fmaf(d[3], u.p.w, -sum.w) / d[3] : 0.0f);
    }
    const double zd[4] = {u.z.x, u.z.y, u.z.z, u.z.w}, pd[4] = {u.p.x, u.p.y, u.p.z, u.p.w}, qd[4] = {qn.x, qn.y, qn.z, qn.w};
    if (inner) {
        double zz = 0.0, pq = 0.0, qz = 0.0, qq = 0.0;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            zz += zd[m] * zd[m];
            pq += pd[m] * qd[m];
            qz += qd[m] * zd[m];
            qq += qd[m] * qd[m];
        }
        v[kRZ] += 6.0 * zz;
        v[kRR] += 36.0 * zz;
        v[kPQ] += 6.0 * pq;
        v[kQZ] += 6.0 * qz;
        v[kRQ] += 36.0 * qz;
        v[kQMQ] += 6.0 * qq;
        v[kQQ] += 36.0 * qq;
    } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const double dm = d[m], r = dm * zd[m], aq = dm * qd[m];
            v[kRZ] += r * zd[m];
            v[kRR] += r * r;
            v[kPQ] += pd[m] * aq;
            v[kQZ] += aq * zd[m];
            v[kRQ] += r * aq;
            v[kQMQ] += aq * qd[m];
            v[kQQ] += aq * aq;
        }
    }
    if (kSmooth && smooth == kSmoothActive) {
        const double sd[4] = {u.s.x, u.s.y, u.s.z, u.s.w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const double dm = d[m];
            v[kCgSums<kSmooth> - 3] += sd[m] * (dm * zd[m]);
            v[kCgSums<kSmooth> - 2] += sd[m] * sd[m];
            v[kCgSums<kSmooth> - 1] += sd[m] * (dm * qd[m]);
        }
    }
    return qn;
}

// Grids too large for the SMs' own memories: a block takes a run of consecutive groups of every plane of a
// slab and marches along z.  p_k of the run and of the row before and after
// it goes to shared memory once per plane; a thread keeps p_k of its own
// groups in the planes below and above.  Each vector is then read once per
// cell (and twice at the runs' and slabs' ends) instead of once per
// neighbour.  The next plane's loads are in flight while a plane is computed.
// Threads own groups of the run with both rows; the rows' are staged only.
template <bool kSmooth, int kPer>
__device__ __forceinline__ void cg_phase_march(const CgArgs& a, const CgStep& k, double (&v)[kCgSums<kSmooth>]) {
    const PadGeom& g = a.g;
    extern __shared__ float4 planes[];  // [3][row | run | row]
    const uint32_t* code4 = reinterpret_cast<const uint32_t*>(a.code);
    const uint32_t halo = g.pitch / 4u, plane_quads = halo * g.ny;
    constexpr uint32_t kSpan = kPer * kCgThreads;
    for (uint32_t item = blockIdx.x; item < a.runs * a.slabs; item += gridDim.x) {
        const uint32_t first = (item % a.runs) * a.run, count = min(a.run, plane_quads - first);
        const int z0 = static_cast<int>(item / a.runs * a.slab), z1 = min(z0 + static_cast<int>(a.slab), static_cast<int>(g.nz));
        const uint32_t origin = g.base + 4u * first - g.pitch + 4u * threadIdx.x;
        bool staged[kPer], owned[kPer];
#pragma unroll
        for (int m = 0; m < kPer; ++m) {
            const uint32_t t = threadIdx.x + m * kCgThreads;
            staged[m] = t < count + 2u * halo;
            owned[m] = t >= halo && t < halo + count;
        }
        CgLoad next[kPer];
        float4 next_e[kPer];
        uint32_t next_c[kPer];
        CgQuad u[2][kPer];  // planes z and z + 1
        float4 below[kPer];
        auto fetch = [&](int z) {
            const uint32_t at = origin + g.plane * static_cast<uint32_t>(z);
            const bool inside = z >= z0 && z < z1;
#pragma unroll
            for (int m = 0; m < kPer; ++m) {
                const uint32_t i = at + 4u * m * kCgThreads;
                if (inside ? staged[m] : owned[m]) next[m] = cg_load(k, i);
                if (inside && owned[m]) {
                    next_e[m] = ld4(a.e + i);
                    next_c[m] = code4[i / 4u];
                }
            }
        };
        // the fetched plane's p_k into shared memory, its z, p, e out
        auto stage = [&](int z, CgQuad (&w)[kPer]) {
            float4* s = planes + static_cast<uint32_t>((z + 3) % 3) * kSpan + threadIdx.x;
            const uint32_t at = origin + g.plane * static_cast<uint32_t>(z);
            const bool inside = z >= z0 && z < z1;
#pragma unroll
            for (int m = 0; m < kPer; ++m) {
                w[m].z = axpy4(next[m].z, -k.alpha, next[m].q);
                w[m].p = axpy4(w[m].z, k.beta, next[m].p);
                if (!inside) continue;
                if (staged[m]) s[m * kCgThreads] = w[m].p;
                if (owned[m]) {
                    w[m].c4 = next_c[m];
                    cg_begin<kSmooth>(a, k, at + 4u * m * kCgThreads, next[m], next_e[m], w[m]);
                }
            }
        };
        __syncthreads();  // the item before is done with the planes
        fetch(z0 - 1);
        stage(z0 - 1, u[0]);
#pragma unroll
        for (int m = 0; m < kPer; ++m) below[m] = u[0][m].p;
        fetch(z0);
        stage(z0, u[0]);
        fetch(z0 + 1);
#pragma unroll 1
        for (int z = z0; z < z1; ++z) {
            stage(z + 1, u[1]);
            __syncthreads();  // plane z is complete; everyone is past plane z - 1
            if (z + 1 < z1) fetch(z + 2);
            const float4* s = planes + static_cast<uint32_t>((z + 3) % 3) * kSpan + threadIdx.x;
            const uint32_t at = origin + g.plane * static_cast<uint32_t>(z);
#pragma unroll
            for (int m = 0; m < kPer; ++m) {
                if (owned[m]) {
                    const float4* here = s + m * kCgThreads;
                    const float4 c = u[0][m].p, lo = *(here - halo), hi = *(here + halo), up = u[1][m].p, down = below[m];
                    const float left = reinterpret_cast<const float*>(here)[-1], right = reinterpret_cast<const float*>(here)[4];
                    const float4 sum = make_float4(left + c.y + lo.x + hi.x + down.x + up.x, c.x + c.z + lo.y + hi.y + down.y + up.y,
                                                   c.y + c.w + lo.z + hi.z + down.z + up.z, c.z + right + lo.w + hi.w + down.w + up.w);
                    if (u[0][m].c4 & kCodeReal4) {
                        const float4 q = cg_operator<kSmooth>(sum, u[0][m], k.smooth, v);
                        store_quad(g, k.qw, at + 4u * m * kCgThreads, u[0][m].c4, q);
                    }
                }
                below[m] = u[0][m].p;
                u[0][m] = u[1][m];
            }
        }
    }
}

// x64 += e_k + alpha p_k of one cell, or with smoothing the smoothed iterate
// of step k + 1: y_k = y + eta (e - y), then y_k + eta_next (e + alpha p - y_k).
struct CgFold {
    float alpha;
    bool smoothed;
    double eta, eta_next;
    __device__ __forceinline__ double step(float e, float p, float y0) const {
        const double x = static_cast<double>(e) + static_cast<double>(alpha) * static_cast<double>(p);
        if (!smoothed) return x;
        const double y = static_cast<double>(y0) + eta * (static_cast<double>(e) - static_cast<double>(y0));
        return y + eta_next * (x - y);
    }
};

// The marching form's vectors live in memory, padded.
constexpr int kMarchPer = 1;
template <bool kSmooth>
struct MarchForm {
    const CgArgs& a;
    __device__ __forceinline__ void setup() { pad_phase(a); }
    __device__ __forceinline__ void residual(int mode, double (&v)[3], double scale) {
        residual_to(a.c, PadStore{a}, mode, v, scale);
        if (!a.g.periodic) return;
        const PadGeom& g = a.g;  // the copies of p and q start at zero with their cells
        for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < g.total; j += gridDim.x * blockDim.x) {
            const uint32_t row = fastdiv(j, g.dpitch), zz = fastdiv(row, g.drows);
            const uint32_t x = j - row * g.pitch, y = row - zz * g.rows;
            if (x < g.nx && y < g.ny && zz >= 1u && zz <= g.nz) continue;
            a.p[0][j] = 0.0f;
            a.q[0][j] = 0.0f;
        }
    }
    __device__ __forceinline__ void begin_pass() {}
    __device__ __forceinline__ void phase(int k, float alpha, float beta, float eta, int smooth, double (&v)[kCgSums<kSmooth>]) {
        const int from = k & 1, to = from ^ 1;
        const CgStep step{a.z[from], a.p[from], a.q[from], a.z[to], a.p[to], a.q[to], alpha, beta, eta, smooth};
#pragma unroll
        for (int i = 0; i < kCgSums<kSmooth>; ++i) v[i] = 0.0;
        cg_phase_march<kSmooth, kMarchPer>(a, step, v);
    }
    __device__ __forceinline__ void prefetch(int) {}
    __device__ __forceinline__ void fold(int k, const CgFold& f) {
        const uint64_t n = cell_count(a.c.op.g);
        const float* p = a.p[(k + 1) & 1];
        for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
            const uint32_t row = fastdiv(static_cast<uint32_t>(i), a.g.dnx), z = fastdiv(row, a.g.dny);
            const uint32_t j = a.g.base + (static_cast<uint32_t>(i) - row * a.g.nx) + a.g.pitch * (row - z * a.g.ny) + a.g.plane * z;
            a.c.x64[i] += f.step(a.e[j], p[j], f.smoothed ? a.y[j] : 0.0f);
        }
    }
};

// --------------------------------------------------------- resident form
// Grids whose vectors fit the SMs: each block keeps a brick of whole rows
// (by x bz of them), kPer 4-cell groups per thread, with z, p, q in registers
// and e (with smoothing s, y) in shared memory for the whole pass.  p_k of
// the brick and of the rows around it is laid out in shared memory for the
// operator.  The rows around are advanced by this block as well, from z and p
// kept in shared memory, so that only their q has to come from its owner:
// one 16-byte load per surrounding group and iteration is all that crosses
// the L2 besides the sums.  An iteration is then the reduction, that load's
// latency and about a microsecond of arithmetic.
struct RowStore {  // z alone, rows of 4 row_quads floats, zeros past the row
    const CgArgs& a;
    __device__ __forceinline__ size_t at(int x, int y, int z) const {
        return static_cast<size_t>(x) + 4u * a.brick.row_quads * (static_cast<size_t>(y) + static_cast<size_t>(a.g.ny) * static_cast<size_t>(z));
    }
    __device__ __forceinline__ void quad(int x, int y, int z, const float4& v) const { st4(a.z[0] + at(x, y, z), v); }
    __device__ __forceinline__ void cell(int x, int y, int z, float v) const {
        float* p = a.z[0] + at(x, y, z);
        *p = v;
        if (x == static_cast<int>(a.g.nx) - 1)
            for (int j = 1; x + j < static_cast<int>(4u * a.brick.row_quads); ++j) p[j] = 0.0f;
    }
};

constexpr size_t brick_smem(uint32_t row_quads, uint32_t by, uint32_t bz, int per, bool smooth) {
    return sizeof(float4) * (1ull + (bz + 2ull) * (by + 2ull) * (row_quads + 1ull) + static_cast<size_t>(per) * kCgThreads * (smooth ? 5 : 3));
}

template <bool kSmooth, int kPer>
struct ResidentForm {
    const CgArgs& a;
    float4 z[kPer], p[kPer], q[kPer], halo_q[kPer];
    uint32_t cell_at[kPer];  // the group's first float in a row vector
    uint32_t box_at[kPer];   // its place in the brick's box
    uint32_t code[kPer];     // codes of its cells (0: no group)
    uint32_t halo_at[kPer], halo_box[kPer];
    float4 *box, *mine;      // shared memory: p of the brick and around; e, s, y, surrounding z and p by thread
    uint32_t line, sheet;    // box strides, in groups: y and z
    bool rim[kPer];          // other blocks read the group's q
    static constexpr uint32_t kNone = 0xffffffffu;

    __device__ __forceinline__ float4& keep(int what, int m) { return mine[(what * kPer + m) * kCgThreads + threadIdx.x]; }
    enum { kE = 0, kHaloZ = 1, kHaloP = 2, kS = 3, kY = 4 };

    __device__ __forceinline__ void setup() {
        extern __shared__ float4 shared[];
        const BrickGeom& b = a.brick;
        const PadGeom& g = a.g;
        const uint32_t width = b.row_quads;
        box = shared;
        line = width + 1u;
        sheet = line * (b.by + 2u);
        const uint32_t box_quads = 1u + sheet * (b.bz + 2u);
        mine = shared + box_quads;
        for (uint32_t i = threadIdx.x; i < box_quads; i += kCgThreads) box[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const uint32_t y0 = (blockIdx.x % b.bricks_y) * b.by, z0 = (blockIdx.x / b.bricks_y) * b.bz;
        const uint32_t ny = min(b.by, g.ny - y0), nz = min(b.bz, g.nz - z0);
        auto box_index = [&](int y, int zz, uint32_t gx) { return 1u + static_cast<uint32_t>(zz + 1) * sheet + static_cast<uint32_t>(y + 1) * line + gx; };
#pragma unroll
        for (int m = 0; m < kPer; ++m) {
            const uint32_t t = threadIdx.x + m * kCgThreads;
            const uint32_t row = t / width, gx = t - row * width, ry = row % ny, rz = row / ny;
            code[m] = 0u;
            rim[m] = false;
            box_at[m] = cell_at[m] = 0u;
            if (rz < nz) {
                const int y = static_cast<int>(y0 + ry), zz = static_cast<int>(z0 + rz);
                cell_at[m] = 4u * (gx + width * (static_cast<uint32_t>(y) + g.ny * static_cast<uint32_t>(zz)));
                box_at[m] = box_index(static_cast<int>(ry), static_cast<int>(rz), gx);
                rim[m] = ry == 0u || ry == ny - 1u || rz == 0u || rz == nz - 1u;
                for (int l = 0; l < 4; ++l) {
                    const int x = static_cast<int>(4u * gx) + l;
                    if (x >= static_cast<int>(g.nx)) break;
                    CellStencil s;
                    const bool act = stencil(a.c.op, x, y, zz, idx3(x, y, zz, static_cast<int>(g.nx), static_cast<int>(g.ny)), s);
                    code[m] |= (kCodeReal | (act ? static_cast<uint32_t>(s.diag) : 0u)) << (8 * l);
                }
            }
            // the rows around: below and above in y (nz each), then in z (ny each)
            halo_at[m] = kNone;
            halo_box[m] = 0u;
            int hy = 0, hz = 0;
            bool there = true;
            if (row < nz) { hy = -1; hz = static_cast<int>(row); }
            else if (row < 2u * nz) { hy = static_cast<int>(ny); hz = static_cast<int>(row - nz); }
            else if (row < 2u * nz + ny) { hy = static_cast<int>(row - 2u * nz); hz = -1; }
            else if (row < 2u * nz + 2u * ny) { hy = static_cast<int>(row - 2u * nz - ny); hz = static_cast<int>(nz); }
            else there = false;
            if (there) {
                int y = static_cast<int>(y0) + hy, zz = static_cast<int>(z0) + hz;
                if (y < 0 || y >= static_cast<int>(g.ny)) { if (g.periodic & 2u) y = y < 0 ? static_cast<int>(g.ny) - 1 : 0; else there = false; }
                if (zz < 0 || zz >= static_cast<int>(g.nz)) { if (g.periodic & 4u) zz = zz < 0 ? static_cast<int>(g.nz) - 1 : 0; else there = false; }
                if (there) {
                    halo_at[m] = 4u * (gx + width * (static_cast<uint32_t>(y) + g.ny * static_cast<uint32_t>(zz)));
                    halo_box[m] = box_index(hy, hz, gx);
                }
            }
        }
        __syncthreads();
    }

    __device__ __forceinline__ void residual(int mode, double (&v)[3], double scale) { residual_to(a.c, RowStore{a}, mode, v, scale); }

    // z of the brick and of the rows around it, everything else zero
    __device__ __forceinline__ void begin_pass() {
        const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int m = 0; m < kPer; ++m) {
            z[m] = code[m] ? ld4(a.z[0] + cell_at[m]) : zero4;
            p[m] = q[m] = halo_q[m] = zero4;
            keep(kE, m) = zero4;
            keep(kHaloP, m) = zero4;
            if (halo_at[m] != kNone) keep(kHaloZ, m) = ld4(a.z[0] + halo_at[m]);
        }
    }

    // The surrounding q of iteration k - 1, as soon as it is complete.
    __device__ __forceinline__ void prefetch(int k) {
        const float* from = a.q[(k - 1) & 1];
#pragma unroll
        for (int m = 0; m < kPer; ++m)
            if (halo_at[m] != kNone) halo_q[m] = ld4(from + halo_at[m]);
    }

    __device__ __forceinline__ void phase(int k, float alpha, float beta, float eta, int smooth, double (&v)[kCgSums<kSmooth>]) {
#pragma unroll
        for (int i = 0; i < kCgSums<kSmooth>; ++i) v[i] = 0.0;
        float4 sm[kPer];
#pragma unroll
        for (int m = 0; m < kPer; ++m) {
            if (halo_at[m] != kNone) {
                const float4 hz = axpy4(keep(kHaloZ, m), -alpha, halo_q[m]);
                const float4 hp = axpy4(hz, beta, keep(kHaloP, m));
                keep(kHaloZ, m) = hz;
                keep(kHaloP, m) = hp;
                box[halo_box[m]] = hp;
            }
            if (code[m] == 0u) continue;
            const float4 zold = z[m], eo = keep(kE, m), en = axpy4(eo, alpha, p[m]);
            keep(kE, m) = en;
            z[m] = axpy4(zold, -alpha, q[m]);
            p[m] = axpy4(z[m], beta, p[m]);
            box[box_at[m]] = p[m];
            if (kSmooth && smooth != kSmoothOff) {
                float d[4];
                cg_diagonal(code[m], d);
                float4 yn = en;
                if (smooth == kSmoothStart) {
                    sm[m] = make_float4(z[m].x * d[0], z[m].y * d[1], z[m].z * d[2], z[m].w * d[3]);
                } else {
                    const float4 so = keep(kS, m), yo = keep(kY, m);
                    sm[m] = make_float4(fmaf(eta, fmaf(zold.x, d[0], -so.x), so.x), fmaf(eta, fmaf(zold.y, d[1], -so.y), so.y),
                                        fmaf(eta, fmaf(zold.z, d[2], -so.z), so.z), fmaf(eta, fmaf(zold.w, d[3], -so.w), so.w));
                    yn = make_float4(fmaf(eta, eo.x - yo.x, yo.x), fmaf(eta, eo.y - yo.y, yo.y), fmaf(eta, eo.z - yo.z, yo.z),
                                     fmaf(eta, eo.w - yo.w, yo.w));
                }
                keep(kS, m) = sm[m];
                keep(kY, m) = yn;
            }
        }
        __syncthreads();
        float* to = a.q[k & 1];
#pragma unroll
        for (int m = 0; m < kPer; ++m) {
            if (code[m] == 0u) continue;
            const float4* here = box + box_at[m];
            const float4 c = p[m], y0 = *(here - line), y1 = *(here + line), z0 = *(here - sheet), z1 = *(here + sheet);
            const float left = reinterpret_cast<const float*>(here)[-1], right = reinterpret_cast<const float*>(here)[4];
            float4 sum = make_float4(left + c.y + y0.x + y1.x + z0.x + z1.x, c.x + c.z + y0.y + y1.y + z0.y + z1.y,
                                     c.y + c.w + y0.z + y1.z + z0.z + z1.z, c.z + right + y0.w + y1.w + z0.w + z1.w);
            if (a.g.periodic & 1u) wrap_row(m, sum);
            CgQuad u;
            u.z = z[m];
            u.p = c;
            if (kSmooth && smooth == kSmoothActive) u.s = sm[m];
            u.c4 = code[m];
            q[m] = cg_operator<kSmooth>(sum, u, smooth, v);
            if (rim[m]) st4(to + cell_at[m], q[m]);
        }
    }

    // The x neighbours across a periodic row's ends (the slot before a row and
    // the slots past it hold zeros).
    __device__ __forceinline__ void wrap_row(int m, float4& sum) const {
        const uint32_t nx = a.g.nx, x0 = cell_at[m] % (4u * a.brick.row_quads), first = box_at[m] - x0 / 4u;
        const float* row = reinterpret_cast<const float*>(box + first);
        if (x0 == 0u) sum.x += row[nx - 1u];
        if (nx - x0 <= 4u) {
            const uint32_t l = nx - 1u - x0;
            const float w = row[0];
            sum.x += l == 0u ? w : 0.0f;
            sum.y += l == 1u ? w : 0.0f;
            sum.z += l == 2u ? w : 0.0f;
            sum.w += l == 3u ? w : 0.0f;
        }
    }

    __device__ __forceinline__ void fold(int, const CgFold& f) {
#pragma unroll
        for (int m = 0; m < kPer; ++m) {
            if (code[m] == 0u) continue;
            const uint32_t width = 4u * a.brick.row_quads, row = cell_at[m] / width, x0 = cell_at[m] - row * width;
            const float4 e = keep(kE, m);
            float4 y = e;
            if (kSmooth && f.smoothed) y = keep(kY, m);
            const float ev[4] = {e.x, e.y, e.z, e.w}, pv[4] = {p[m].x, p[m].y, p[m].z, p[m].w}, yv[4] = {y.x, y.y, y.z, y.w};
            double* x = a.c.x64 + static_cast<size_t>(row) * a.g.nx + x0;
#pragma unroll
            for (int l = 0; l < 4; ++l)
                if (x0 + l < a.g.nx) x[l] += f.step(ev[l], pv[l], yv[l]);
        }
    }
};

// ---------------------------------------------------------------- the solve
template <bool kSmooth, class Form>
__device__ __forceinline__ void cg_solve(const CgArgs& a, Form form) {
    const PcgArgs& c = a.c;
    SolverState* st = c.st;
    SlotSync sync{a.slots, st, 0ull};
    double v3[3];
    double scale = c.guess ? 1.0 : 0.0;
    if (c.guess && c.scale_guess) {
        double e2[2];
        guess_energy_phase(c, e2);
        if (!slot_reduce(sync, e2)) return;
        scale = (e2[1] > 0.0 && isfinite(e2[0] / e2[1])) ? e2[0] / e2[1] : 0.0;
    }
    form.setup();
    form.residual(c.guess ? kFromGuess : kFromZero, v3, scale);
    if (!slot_reduce(sync, v3)) return;
    const double bb = v3[0];
    double rr = v3[1];
    uint32_t warm = c.guess ? 1u : 0u;
    if (c.guess && !(rr <= bb)) {  // the guess is worse than zero: fall back
        warm = 0u;
        scale = 0.0;
        form.residual(kFromZero, v3, 1.0);
        if (!slot_reduce(sync, v3)) return;
        rr = v3[1];
    }
    const double initial = bb > 0.0 ? sqrt(rr / bb) : 0.0;
    const double target2 = c.tol * c.tol * bb;
    // (when and from where smoothing pays: see pcg_kernel)
    const bool smooth_run = kSmooth && warm != 0u && rr < 0.01 * bb;
    const double smooth_begin2 = 100.0 * target2;
    uint32_t iterations = 0, refinements = 0, smoothed_iterations = 0;
    uint32_t status = XS_OK;
    while (true) {
        if (!(rr <= target2)) {
            if (!isfinite(rr)) { status = XS_NUMERICAL_ERROR; break; }
            if (iterations >= c.max_iterations || refinements > kMaxRefinements) { status = XS_NOT_CONVERGED; break; }
        } else {
            status = XS_OK;
            break;
        }
        form.begin_pass();
        int k = 0;
        float alpha = 0.0f, beta = 0.0f;
        double eta = 0.0, eta_next = 0.0;
        bool broke = false, smoothed = false;
        int smode = smooth_run && rr < smooth_begin2 ? kSmoothStart : kSmoothOff;
        while (true) {
            double v[kCgSums<kSmooth>];
            form.phase(k, alpha, beta, static_cast<float>(eta), smode, v);
            if (!slot_reduce(sync, v)) return;
            form.prefetch(k + 1);
            if (!(v[kPQ] > 0.0) || !isfinite(v[kPQ])) { broke = true; break; }
            alpha = static_cast<float>(v[kRZ] / v[kPQ]);
            const double al = alpha;
            const double rz_next = v[kRZ] - 2.0 * al * v[kQZ] + al * al * v[kQMQ];
            const double rr_next = v[kRR] - 2.0 * al * v[kRQ] + al * al * v[kQQ];
            ++iterations;
            if (smode != kSmoothOff) ++smoothed_iterations;
            if (!isfinite(rr_next)) { broke = true; break; }
            // rz_next <= 0: the step has reached the rounding of its sums
            const bool done = rr_next <= target2 || !(rz_next > 0.0) || iterations >= c.max_iterations;
            beta = static_cast<float>(rz_next / v[kRZ]);
            if (kSmooth && smode != kSmoothOff) {
                // sums of s_{k-1} against r_k, itself and A p_k -> eta_k, then of s_k against r_{k+1} -> eta_{k+1}
                double sr = v[kRR], ss = v[kRR], sq = v[kRQ];
                if (smode == kSmoothActive) {
                    sr = v[kCgSums<kSmooth> - 3];
                    ss = v[kCgSums<kSmooth> - 2];
                    sq = v[kCgSums<kSmooth> - 1];
                    const double den = v[kRR] - 2.0 * sr + ss;
                    eta = den > 0.0 ? (ss - sr) / den : 0.0;
                    ss += 2.0 * eta * (sr - ss) + eta * eta * den;
                    sr += eta * (v[kRR] - sr);
                    sq += eta * (v[kRQ] - sq);
                } else {
                    eta = 0.0;
                }
                const double sr_next = sr - al * sq;
                const double den = rr_next - 2.0 * sr_next + ss;
                eta_next = den > 0.0 ? (ss - sr_next) / den : 0.0;
                const double ss_next = ss + 2.0 * eta_next * (sr_next - ss) + eta_next * eta_next * den;
                if (!done && ss_next <= target2 && isfinite(ss_next)) {
                    smoothed = true;
                    break;
                }
                smode = kSmoothActive;
            } else if (smooth_run && rr_next < smooth_begin2) {
                smode = kSmoothStart;
            }
            if (done) break;
            ++k;
        }
        if (broke) {
            status = XS_NUMERICAL_ERROR;
            break;
        }
        form.fold(k, CgFold{alpha, smoothed, eta, eta_next});
        double none[1] = {0.0};
        if (!slot_reduce(sync, none)) return;
        form.residual(kFromX64, v3, 1.0);
        if (!slot_reduce(sync, v3)) return;
        rr = v3[1];
        ++refinements;
    }
    if (status != XS_OK && rr <= target2) status = XS_OK;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->stats.iterations = iterations;
        st->stats.status = status;
        st->stats.refinements = refinements;
        st->stats.warm_start_used = warm;
        st->stats.rhs_norm = sqrt(bb);
        st->stats.initial_residual = initial;
        st->stats.final_residual = bb > 0.0 ? sqrt(rr / bb) : 0.0;
        st->stats.guess_scale = scale;
        st->stats.smoothed_iterations = smoothed_iterations;
    }
}

// kPer: groups per thread of the resident form; 0: the marching form.
template <bool kSmooth, int kPer>
__global__ void __launch_bounds__(kCgThreads, 1) cg_kernel(const __grid_constant__ CgArgs a) {
    if constexpr (kPer == 0) cg_solve<kSmooth>(a, MarchForm<kSmooth>{a});
    else cg_solve<kSmooth>(a, ResidentForm<kSmooth, kPer>{a});
}

}  // namespace xs
