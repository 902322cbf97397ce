// Red-black Gauss-Seidel with the whole grid in the SMs (included by
// pressure.cu): the reference's sweeps (operators.cu:885-902, 1004-1013) with
// the same sums in the same order, so the same bits.
//
// Each block keeps a brick of whole rows.  A row's cells lie split by colour,
// so that a half sweep reads the other colour's values contiguously: cell x of
// row (y, z) is entry m of colour c, x = 2 m + ((y + z + c) & 1), and its x
// neighbours are entries m and m - 1 (even start) or m + 1 (odd start) of the
// other colour.  Pressures are in shared memory, with a row of surrounding
// values on each side; right-hand sides and diagonals are in registers, kPer
// groups of 4 entries per thread and colour.  Slots beyond the grid hold what
// the sum adds there: 0 for a zero-gradient face, the value of a fixed one.
//
// After each half sweep a block passes on only the colour it just wrote, of
// its outermost rows, and waits only for the (at most four) bricks it borders:
// one flag each.  A block can be no more than one half sweep ahead of a
// neighbour, which is why one copy of the outermost rows suffices: they are
// written again two half sweeps later, after the neighbour's flag for the one
// between.
//
// What bounds it: the shared memory (28 wavefronts per 128 cells, about 1.2 us
// for a block of 128 x 192 x 128) and the neighbours' flags and rows (about 2
// us) per half sweep.  The general kernel looks every neighbour up in memory,
// half of its threads idle.  160 sweeps, general -> resident: 64^3 2.82 -> 0.74
// ms, 128x192x128 12.0 -> 1.73 (with colliders 15.9 -> 1.80), 100 sweeps of
// 256x128x64 5.71 -> 0.94.
#pragma once

namespace xs {

struct RbgsBrick {
    uint32_t quads;          // groups of 4 entries per row and colour
    uint32_t by, bz;         // rows of a brick
    uint32_t bricks_y, bricks_z;
};

struct RbgsResidentArgs {
    RbgsArgs c;
    RbgsBrick b;
    float* rim[2];           // outermost rows of each colour: 4 quads floats per row of the grid
    uint32_t* flags;         // half sweeps done, one per block, 64 bytes apart
};

constexpr int kRbgsThreads = 512;
constexpr uint32_t kRbgsFlagStride = 16;
constexpr size_t rbgs_smem(const RbgsBrick& b) {
    return sizeof(float4) * 2ull * (1ull + (b.by + 2ull) * (b.bz + 2ull) * (b.quads + 1ull));
}

__device__ __forceinline__ float rbgs_cell(float rhs, float l, float r, float d, float u, float b, float f, uint32_t diag, float old) {
    // neighbour order of the reference: -x, +x, -y, +y, -z, +z
    float sum = rhs + l;
    sum += r;
    sum += d;
    sum += u;
    sum += b;
    sum += f;
    return diag == 0u ? old : sum / static_cast<float>(diag);
}

template <int kPer>
__global__ void __launch_bounds__(kRbgsThreads, 1) rbgs_resident_kernel(const __grid_constant__ RbgsResidentArgs a) {
    extern __shared__ float4 box[];
    __shared__ double red[4 * 32];
    __shared__ unsigned failed;
    const Operator& op = a.c.op;
    const Grid& g = op.g;
    const RbgsBrick& b = a.b;
    const uint32_t width = b.quads, line = 4u * (width + 1u), sheet = line * (b.by + 2u);
    const uint32_t half = 4u + sheet * (b.bz + 2u);  // floats of one colour
    float* const p0 = reinterpret_cast<float*>(box);
    const uint32_t brick_y = blockIdx.x % b.bricks_y, brick_z = blockIdx.x / b.bricks_y;
    const int y0 = static_cast<int>(brick_y * b.by), z0 = static_cast<int>(brick_z * b.bz);
    const int ny = min(static_cast<int>(b.by), g.ny - y0), nz = min(static_cast<int>(b.bz), g.nz - z0);
    auto row_at = [&](int ry, int rz) { return 4u + static_cast<uint32_t>(rz + 1) * sheet + static_cast<uint32_t>(ry + 1) * line; };
    auto fixed_value = [&](int face) { return op.pb.modes[face] == 0u ? op.pb.values[face] : 0.0f; };
    // start values: 0 in the grid, the boundary's part beyond it
    for (uint32_t i = threadIdx.x; i < half; i += kRbgsThreads) {
        const int j = static_cast<int>(i) - 4;  // (the lone first group: x = -1 of a row no cell reads)
        const int rz = j < 0 ? -1 : j / static_cast<int>(sheet) - 1, rest = j < 0 ? 0 : j % static_cast<int>(sheet);
        const int ry = rest / static_cast<int>(line) - 1, m = rest % static_cast<int>(line);
        // the last slot of a row is entry -1 of the next one
        const bool before = m == static_cast<int>(line) - 1;
        const int yr = before ? ry + 1 : ry;
        for (int c = 0; c < 2; ++c) {
            const int y = y0 + yr, z = z0 + rz;
            const int x = 2 * (before ? -1 : m) + ((y + z + c) & 1);
            float v = 0.0f;
            if (z < 0) v = fixed_value(4);
            else if (z >= g.nz) v = fixed_value(5);
            else if (y < 0) v = fixed_value(2);
            else if (y >= g.ny) v = fixed_value(3);
            else if (x == -1) v = fixed_value(0);
            else if (x == g.nx) v = fixed_value(1);
            p0[c * half + i] = v;
        }
    }
    float rhs[2][kPer][4];
    uint32_t diag[2][kPer];       // a byte per entry, 0: left as it is
    uint32_t at[kPer], rim_at[kPer];
    uint32_t flags = 0u;          // bits 2m, 2m + 1: group m exists, is in an outermost row; bit 16 + m: parity of y + z
#pragma unroll
    for (int m = 0; m < kPer; ++m) {
        const uint32_t t = threadIdx.x + m * kRbgsThreads, row = t / width, q = t - row * width;
        const int ry = static_cast<int>(row % static_cast<uint32_t>(ny)), rz = static_cast<int>(row / static_cast<uint32_t>(ny));
        at[m] = rim_at[m] = 0u;
        diag[0][m] = diag[1][m] = 0u;
        if (rz >= nz) continue;
        const int y = y0 + ry, z = z0 + rz, parity = (y + z) & 1;
        at[m] = row_at(ry, rz) + 4u * q;
        rim_at[m] = 4u * (q + width * (static_cast<uint32_t>(y) + static_cast<uint32_t>(g.ny) * static_cast<uint32_t>(z)));
        flags |= 1u << (2 * m);
        if (ry == 0 || ry == ny - 1 || rz == 0 || rz == nz - 1) flags |= 2u << (2 * m);
        if (parity) flags |= 1u << (16 + m);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int x = static_cast<int>(8u * q) + e, c = (e & 1) ^ parity;
            float r = 0.0f;
            uint32_t d = 0u;
            if (x < g.nx) {
                const uint64_t i = idx3(x, y, z, g.nx, g.ny);
                CellStencil s;
                if (stencil(op, x, y, z, i, s)) d = static_cast<uint32_t>(s.diag);
                r = a.c.rhs[i];
            }
            // (c is a run-time value: select, so that the arrays stay in registers)
            if (c == 0) { rhs[0][m][e >> 1] = r; diag[0][m] |= d << (8 * (e >> 1)); }
            else { rhs[1][m][e >> 1] = r; diag[1][m] |= d << (8 * (e >> 1)); }
        }
    }
    __syncthreads();
    const int me = static_cast<int>(blockIdx.x);
    // the flag this thread watches: its block's neighbours below and above in y and z
    int watch = -1;
    if (threadIdx.x == 0 && brick_y > 0) watch = me - 1;
    if (threadIdx.x == 1 && brick_y + 1 < b.bricks_y) watch = me + 1;
    if (threadIdx.x == 2 && brick_z > 0) watch = me - static_cast<int>(b.bricks_y);
    if (threadIdx.x == 3 && brick_z + 1 < b.bricks_z) watch = me + static_cast<int>(b.bricks_y);
    const uint32_t around = 2u * static_cast<uint32_t>(ny + nz) * width;
    if (threadIdx.x == 0) failed = 0u;
    __syncthreads();
    for (uint32_t step = 0; step < 2u * a.c.sweeps; ++step) {
        const int c = static_cast<int>(step & 1u);
        float* mine = p0 + c * half;
        float* other = p0 + (c ^ 1) * half;
        if (step > 0) {  // the neighbours' outermost rows of the other colour
            if (watch >= 0) {
                const uint32_t* flag = a.flags + static_cast<size_t>(watch) * kRbgsFlagStride;
                const long long t0 = clock64();
                uint32_t seen;
                do {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(flag) : "memory");
                    if (seen < step && clock64() - t0 > kBarrierTimeoutCycles) {
                        atomicExch(&a.c.st->error, 1u);
                        failed = 1u;
                        break;
                    }
                } while (seen < step);
            }
            __syncthreads();
            if (failed) return;
            for (uint32_t t = threadIdx.x; t < around; t += kRbgsThreads) {
                const uint32_t row = t / width, q = t - row * width;
                int ry, rz;
                if (row < 2u * static_cast<uint32_t>(nz)) {
                    ry = row < static_cast<uint32_t>(nz) ? -1 : ny;
                    rz = static_cast<int>(row) - (row < static_cast<uint32_t>(nz) ? 0 : nz);
                } else {
                    const int r = static_cast<int>(row) - 2 * nz;
                    rz = r < ny ? -1 : nz;
                    ry = r - (r < ny ? 0 : ny);
                }
                const int y = y0 + ry, z = z0 + rz;
                if (y < 0 || y >= g.ny || z < 0 || z >= g.nz) continue;
                const float4* from = reinterpret_cast<const float4*>(
                    a.rim[c ^ 1] + 4u * (q + width * (static_cast<uint32_t>(y) + static_cast<uint32_t>(g.ny) * static_cast<uint32_t>(z))));
                *reinterpret_cast<float4*>(other + row_at(ry, rz) + 4u * q) = __ldcg(from);
            }
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < kPer; ++m) {
            if (!((flags >> (2 * m)) & 1u)) continue;
            const float* o = other + at[m];
            const float4 same = *reinterpret_cast<const float4*>(o);
            const float4 yl = *reinterpret_cast<const float4*>(o - line), yh = *reinterpret_cast<const float4*>(o + line);
            const float4 zl = *reinterpret_cast<const float4*>(o - sheet), zh = *reinterpret_cast<const float4*>(o + sheet);
            const float4 old = *reinterpret_cast<const float4*>(mine + at[m]);
            // this colour starts at x = 0 or x = 1 of the row
            const bool odd = (((flags >> (16 + m)) & 1u) ^ static_cast<uint32_t>(c)) != 0u;
            const float edge = odd ? o[4] : o[-1];
            const float l0 = odd ? same.x : edge, l1 = odd ? same.y : same.x, l2 = odd ? same.z : same.y, l3 = odd ? same.w : same.z;
            const float r0 = odd ? same.y : same.x, r1 = odd ? same.z : same.y, r2 = odd ? same.w : same.z, r3 = odd ? edge : same.w;
            const uint32_t d = c == 0 ? diag[0][m] : diag[1][m];
            float4 v;
            v.x = rbgs_cell(c == 0 ? rhs[0][m][0] : rhs[1][m][0], l0, r0, yl.x, yh.x, zl.x, zh.x, d & 255u, old.x);
            v.y = rbgs_cell(c == 0 ? rhs[0][m][1] : rhs[1][m][1], l1, r1, yl.y, yh.y, zl.y, zh.y, (d >> 8) & 255u, old.y);
            v.z = rbgs_cell(c == 0 ? rhs[0][m][2] : rhs[1][m][2], l2, r2, yl.z, yh.z, zl.z, zh.z, (d >> 16) & 255u, old.z);
            v.w = rbgs_cell(c == 0 ? rhs[0][m][3] : rhs[1][m][3], l3, r3, yl.w, yh.w, zl.w, zh.w, d >> 24, old.w);
            *reinterpret_cast<float4*>(mine + at[m]) = v;
            if ((flags >> (2 * m)) & 2u) *reinterpret_cast<float4*>(a.rim[c] + rim_at[m]) = v;
        }
        __syncthreads();  // every outermost row is written
        if (threadIdx.x == 0) {
            asm volatile("fence.acq_rel.gpu;\n st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(a.flags + static_cast<size_t>(me) * kRbgsFlagStride), "r"(step + 1u)
                         : "memory");
        }
    }
    // the pressure, both colours back in order
#pragma unroll
    for (int m = 0; m < kPer; ++m) {
        if (!((flags >> (2 * m)) & 1u)) continue;
        const float4 c0 = *reinterpret_cast<const float4*>(p0 + at[m]), c1 = *reinterpret_cast<const float4*>(p0 + half + at[m]);
        const bool odd = ((flags >> (16 + m)) & 1u) != 0u;
        const float4 e = odd ? c1 : c0, o = odd ? c0 : c1;  // entries at even and at odd x
        const float v[8] = {e.x, o.x, e.y, o.y, e.z, o.z, e.w, o.w};
        const uint32_t row = rim_at[m] / (4u * width), q = rim_at[m] / 4u - row * width;
        float* out = a.c.p + static_cast<size_t>(row) * static_cast<size_t>(g.nx) + 8u * q;
#pragma unroll
        for (int x = 0; x < 8; ++x)
            if (static_cast<int>(8u * q) + x < g.nx) out[x] = v[x];
    }
    if (!grid_barrier(a.c.st, a.c.partials, red)) return;
    rbgs_report(a.c, red);
}

}  // namespace xs
