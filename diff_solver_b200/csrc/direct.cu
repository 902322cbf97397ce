// Direct solve of the pressure system on the fluid grid itself, in FP32, as
// the start of a warm-started PCG solve.
//
// Without colliders the operator is the Kronecker sum of three 1D operators
// (spectral.cu).  Two axes are transformed to their eigenbases, and along the
// third a tridiagonal system remains for every pair of modes:
//
//     (lambda_a + lambda_b) x_j + (T x)_j = b_j .
//
// Four transforms and one tridiagonal pass instead of rounds of sweeps,
// restriction, coarse solve, interpolation and a line step, and what is left
// of the residual is rounding noise, which the PCG that follows removes in a
// few iterations.
//
// Transforms.  The 1D bases of an axis with equal ends, or a periodic one
// (sampled half a cell off, cos and sin of 2 pi m (j + 1/2) / n), are even or
// odd under j -> n - 1 - j: a line is folded into sums and differences of
// mirrored values, and even and odd modes are two products of half the size,
// half the operations of a full basis.  An axis with unequal ends (the
// plume's open top) has no such symmetry: it is the one left tridiagonal.
//
// What bounds it: the products, n operations per cell and transform on the FP32
// pipes (256^3: 4.3 GFLOP in 122 us, 35 TFLOP/s of the 71 that packed products
// reach with their operands in registers), the tridiagonal pass by memory and
// its exponentials (75 us).  One solve: 128^3 80 us, 256^3 0.58 ms, 512x512x256
// 3.1 ms.  What it replaces there, start and fine solve together (early plume):
// 128^3 1.0 -> 0.21 ms, 256^3 with the network 18 -> 1.9 ms, 512x512x256 50 ->
// 7.1 ms, with no iteration left to do from two solves (see direct_start).
#include <algorithm>

#include "launch.cuh"
#include "pressure.cuh"

namespace xs {

namespace {

enum FoldKind : int { kFoldZero = 0, kFoldFixed = 1, kFoldPeriodic = 2 };  // both ends zero-gradient / fixed value, or wrapped

constexpr int P = kDirectMax / 2;  // most modes of one symmetry

// Mode i of an axis in the order used here: the even modes 0 .. h - 1, then
// the odd ones; entry at position j, and eigenvalue, in FP64.
__device__ double fold_entry(int kind, int n, int half, int i, int j) {
    const double dn = n;
    switch (kind) {
        case kFoldZero: {
            const int k = 2 * i + half;
            return (k == 0 ? sqrt(1.0 / dn) : sqrt(2.0 / dn)) * cospi(k * (j + 0.5) / dn);
        }
        case kFoldFixed: return sqrt(2.0 / (dn + 1.0)) * sinpi((2 * i + half + 1.0) * (j + 1.0) / (dn + 1.0));
        default:
            if (half == 0) return (i == 0 ? sqrt(1.0 / dn) : sqrt(2.0 / dn)) * cospi(2.0 * i * (j + 0.5) / dn);
            return (2 * (i + 1) == n ? sqrt(1.0 / dn) : sqrt(2.0 / dn)) * sinpi(2.0 * (i + 1) * (j + 0.5) / dn);
    }
}

__device__ double fold_eigenvalue(int kind, int n, int half, int i) {
    // 2 - 2 cos(t) as 4 sin(t / 2)^2: the smallest ones keep their digits
    const double dn = n;
    const double s = kind == kFoldZero ? sinpi(0.5 * (2 * i + half) / dn)
                                       : (kind == kFoldFixed ? sinpi(0.5 * (2 * i + half + 1.0) / (dn + 1.0)) : sinpi((i + half) / dn));
    return 4.0 * s * s;
}

struct FoldAxes {
    int n[2], kind[2];
};

// Per axis: the even and the odd half of the basis, rows j, columns modes,
// then both transposed; 4 P^2 floats.  Eigenvalues: 2 P per axis.
__global__ void fold_basis_kernel(FoldAxes ax, float* __restrict__ basis, float* __restrict__ eigen) {
    const int a = static_cast<int>(blockIdx.z) >> 1, half = static_cast<int>(blockIdx.z) & 1;
    const int i = static_cast<int>(blockIdx.x * 32 + threadIdx.x), j = static_cast<int>(blockIdx.y * 8 + threadIdx.y);
    const int n = ax.n[a], h = (n + 1) / 2, modes = half ? n / 2 : h;
    if (i >= P || j >= P) return;
    float* m = basis + static_cast<size_t>(a) * 4 * P * P + static_cast<size_t>(half) * P * P;
    const float q = i < modes && j < modes ? static_cast<float>(fold_entry(ax.kind[a], n, half, i, j)) : 0.0f;
    m[j * P + i] = q;
    m[2 * P * P + i * P + j] = q;
    if (j == 0 && i < modes) eigen[a * 2 * P + half * h + i] = static_cast<float>(fold_eigenvalue(ax.kind[a], n, half, i));
}

// ------------------------------------------------------------ transforms
// The lines of one axis: element j of line L of batch b at b * batch_stride +
// L * line_stride + j * stride, one of line_stride and stride being 1.
struct FoldLines {
    int n;
    uint32_t lines;
    uint64_t batch_stride, line_stride, stride;
};

constexpr int kFoldThreads = 256;
constexpr int kFoldLines = 128;  // lines of a tile
constexpr int kFoldModes = 64;   // modes (or positions) of each symmetry of a tile
constexpr int kFoldDepth = 16;   // values of the inner sum staged at a time
constexpr int kFoldPitch = kFoldLines + 4;

struct FoldStage {  // [symmetry]
    float data[2][kFoldDepth][kFoldPitch];
    float mat[2][kFoldDepth][2 * kFoldModes];  // every entry twice, for packed products
};

// Two FP32 fused multiply-adds in one instruction (each rounded as fmaf): a
// tile of sums fed by scalar instructions is held to 51 TFLOP/s by its
// register reads, packed pairs reach the pipes' 71 (measured, operands in
// registers).
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long x, unsigned long long y) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y));
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// One tile of 128 lines by 64 + 64 outputs, 8 lines (two runs of
// 4, so that a warp's 16-byte loads hit every bank once) by 4 + 4 outputs per
// thread (64 sums in registers, 32 packed products against 8 16-byte shared loads
// per step of the inner sum); the next step's operands are loaded while one is multiplied.
// Forward: even and odd coefficients from folded values.  Inverse: s and t
// from even and odd coefficients, x_j = s + t and x_{n-1-j} = s - t.
// kVec: extents and strides that make every run of 4 values along the
// contiguous direction 16-byte aligned.
__device__ __forceinline__ float4 load_run(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_run(const double* p) {
    const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
    return make_float4(static_cast<float>(a.x), static_cast<float>(a.y), static_cast<float>(b.x), static_cast<float>(b.y));
}
__device__ __forceinline__ float4 reversed(const float4& v) { return make_float4(v.w, v.z, v.y, v.x); }

template <bool kInverse, bool kStrided, bool kVec, class Tin>
__global__ void __launch_bounds__(kFoldThreads, 2) fold_transform_kernel(const Tin* __restrict__ in, float* __restrict__ out, FoldLines ls,
                                                                         const float* __restrict__ basis) {
    extern __shared__ __align__(16) unsigned char fold_smem[];
    FoldStage* stage = reinterpret_cast<FoldStage*>(fold_smem);  // [2]
    const int t = static_cast<int>(threadIdx.x), n = ls.n, h = (n + 1) / 2, ho = n / 2;
    const uint32_t L0 = blockIdx.x * kFoldLines;
    const int m0 = static_cast<int>(blockIdx.y) * kFoldModes;
    const uint64_t batch = static_cast<uint64_t>(blockIdx.z) * ls.batch_stride;
    const float* q = basis + (kInverse ? 2 * P * P : 0);
    // A thread's share of a step: kRuns runs of 4 values (of kRuns * 4 single
    // ones) and of their partners -- forward the mirrored values, inverse the
    // odd coefficients -- and one run of each half of the basis.
    constexpr int kRuns = kFoldLines * kFoldDepth / kFoldThreads / 4;
    float4 va[kRuns], vb[kRuns], me, mo;
    // run r: line(s) l and position(s) j; strided runs go along lines, others along j
    auto place = [&](int r, int& l, int& j) {
        const int i = t + r * kFoldThreads;
        if (kStrided) {
            l = 4 * (i % (kFoldLines / 4));
            j = i / (kFoldLines / 4);
        } else {
            l = i / (kFoldDepth / 4);
            j = 4 * (i % (kFoldDepth / 4));
        }
    };
    auto load = [&](int k0) {
#pragma unroll
        for (int r = 0; r < kRuns; ++r) {
            int l, jj;
            place(r, l, jj);
            const int j = k0 + jj;
            const uint32_t L = L0 + l;
            const Tin* line = in + batch + L * ls.line_stride;
            va[r] = vb[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (kVec) {
                if (L >= ls.lines || j >= h) continue;
                va[r] = load_run(line + static_cast<uint64_t>(j) * ls.stride);
                if (kStrided) vb[r] = load_run(line + static_cast<uint64_t>(kInverse ? h + j : n - 1 - j) * ls.stride);
                else vb[r] = kInverse ? load_run(line + h + j) : reversed(load_run(line + n - 4 - j));
            } else {
                float x[4], y[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int je = kStrided ? j : j + e;
                    const uint32_t Le = kStrided ? L + e : L;
                    const Tin* le = kStrided ? line + e : line;  // (strided lines are contiguous)
                    const int other = kInverse ? h + je : n - 1 - je;
                    const bool there = Le < ls.lines && je < h;
                    x[e] = there ? static_cast<float>(le[static_cast<uint64_t>(je) * ls.stride]) : 0.0f;
                    y[e] = there && je < ho ? static_cast<float>(le[static_cast<uint64_t>(other) * ls.stride]) : 0.0f;
                }
                va[r] = make_float4(x[0], x[1], x[2], x[3]);
                vb[r] = make_float4(y[0], y[1], y[2], y[3]);
            }
        }
        // (the basis is padded with zeros to its P x P array)
        const int k = k0 + t / (kFoldModes / 4), c = m0 + 4 * (t % (kFoldModes / 4));
        me = *reinterpret_cast<const float4*>(q + k * P + c);
        mo = *reinterpret_cast<const float4*>(q + P * P + k * P + c);
    };
    auto store = [&](int b) {
#pragma unroll
        for (int r = 0; r < kRuns; ++r) {
            int l, j;
            place(r, l, j);
            float4 x = va[r], y = vb[r];
            if (!kInverse) {
                // an odd line's middle value has no partner: its difference meets zero rows of the odd half
                x = make_float4(va[r].x + vb[r].x, va[r].y + vb[r].y, va[r].z + vb[r].z, va[r].w + vb[r].w);
                y = make_float4(va[r].x - vb[r].x, va[r].y - vb[r].y, va[r].z - vb[r].z, va[r].w - vb[r].w);
            }
            if (kStrided) {
                *reinterpret_cast<float4*>(&stage[b].data[0][j][l]) = x;
                *reinterpret_cast<float4*>(&stage[b].data[1][j][l]) = y;
            } else {
                const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    stage[b].data[0][j + e][l] = xs[e];
                    stage[b].data[1][j + e][l] = ys[e];
                }
            }
        }
        const int k = t / (kFoldModes / 4), c = 4 * (t % (kFoldModes / 4));
        // the first two modes of every thread's four, then the other two: 16-byte runs
        *reinterpret_cast<float4*>(&stage[b].mat[0][k][c]) = make_float4(me.x, me.x, me.y, me.y);
        *reinterpret_cast<float4*>(&stage[b].mat[0][k][kFoldModes + c]) = make_float4(me.z, me.z, me.w, me.w);
        *reinterpret_cast<float4*>(&stage[b].mat[1][k][c]) = make_float4(mo.x, mo.x, mo.y, mo.y);
        *reinterpret_cast<float4*>(&stage[b].mat[1][k][kFoldModes + c]) = make_float4(mo.z, mo.z, mo.w, mo.w);
    };
    // the threads of a warp spread along what is contiguous in the output
    const int tl = kStrided ? t & 15 : t >> 4, tm = kStrided ? t >> 4 : t & 15;
    unsigned long long sums[2][4][4];  // [symmetry][pair of lines][mode]
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) sums[s][i][c] = 0ull;
    load(0);
    store(0);
    __syncthreads();
    for (int k0 = 0, b = 0; k0 < h; k0 += kFoldDepth, b ^= 1) {
        const bool more = k0 + kFoldDepth < h;
        if (more) load(k0 + kFoldDepth);
#pragma unroll
        for (int k = 0; k < kFoldDepth; ++k) {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const ulonglong2 x0 = *reinterpret_cast<const ulonglong2*>(&stage[b].data[s][k][4 * tl]),
                                 x1 = *reinterpret_cast<const ulonglong2*>(&stage[b].data[s][k][kFoldLines / 2 + 4 * tl]);
                const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(&stage[b].mat[s][k][4 * tm]),
                                 w1 = *reinterpret_cast<const ulonglong2*>(&stage[b].mat[s][k][kFoldModes + 4 * tm]);
                const unsigned long long x[4] = {x0.x, x0.y, x1.x, x1.y}, y[4] = {w0.x, w0.y, w1.x, w1.y};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int c = 0; c < 4; ++c) fma2(sums[s][i][c], x[i], y[c]);
            }
        }
        if (more) {
            store(b ^ 1);  // the buffer read one step ago: everyone is past it
            __syncthreads();
        }
    }
    float acc[2][8][4];
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 v = unpack2(sums[s][i][c]);
                acc[s][2 * i][c] = v.x;
                acc[s][2 * i + 1][c] = v.y;
            }
    if (kInverse) {  // x_j = s + o, x_{n-1-j} = s - o
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float s = acc[0][i][c], o = acc[1][i][c];
                acc[0][i][c] = s + o;
                acc[1][i][c] = s - o;
            }
    }
    // outputs of the second half go to n - 1 - m (inverse) or h + m
    if (kVec && kStrided) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int m = m0 + 4 * tm + c;
            if (m >= h) continue;
#pragma unroll
            for (int i = 0; i < 8; i += 4) {
                const uint32_t L = L0 + 4 * tl + (i >> 2) * (kFoldLines / 2);
                if (L >= ls.lines) continue;
                float* line = out + batch + L;
                *reinterpret_cast<float4*>(line + static_cast<uint64_t>(m) * ls.stride) = make_float4(acc[0][i][c], acc[0][i + 1][c], acc[0][i + 2][c], acc[0][i + 3][c]);
                *reinterpret_cast<float4*>(line + static_cast<uint64_t>(kInverse ? n - 1 - m : h + m) * ls.stride) =
                    make_float4(acc[1][i][c], acc[1][i + 1][c], acc[1][i + 2][c], acc[1][i + 3][c]);
            }
        }
        return;
    }
    if (kVec) {
        const int m = m0 + 4 * tm;
        if (m >= h) return;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t L = L0 + 4 * tl + (i & 3) + (i >> 2) * (kFoldLines / 2);
            if (L >= ls.lines) continue;
            float* line = out + L * ls.line_stride;
            const float4 a = make_float4(acc[0][i][0], acc[0][i][1], acc[0][i][2], acc[0][i][3]);
            const float4 b = make_float4(acc[1][i][0], acc[1][i][1], acc[1][i][2], acc[1][i][3]);
            *reinterpret_cast<float4*>(line + m) = a;
            if (kInverse) *reinterpret_cast<float4*>(line + n - 4 - m) = reversed(b);
            else *reinterpret_cast<float4*>(line + h + m) = b;
        }
        return;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int m = m0 + 4 * tm + c;
        if (m >= h) continue;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t L = L0 + 4 * tl + (i & 3) + (i >> 2) * (kFoldLines / 2);
            if (L >= ls.lines) continue;
            float* line = out + batch + L * ls.line_stride;
            line[static_cast<uint64_t>(m) * ls.stride] = acc[0][i][c];
            if (m < ho) line[static_cast<uint64_t>(kInverse ? n - 1 - m : h + m) * ls.stride] = acc[1][i][c];
        }
    }
}

template <bool kInverse, bool kStrided, bool kVec, class Tin>
XsStatus launch_transform(cudaStream_t st, const Tin* in, float* out, const FoldLines& ls, uint32_t batches, const float* basis) {
    static DeviceOnce configured;
    if (!configured.run([] {
            return cudaFuncSetAttribute(fold_transform_kernel<kInverse, kStrided, kVec, Tin>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(2 * sizeof(FoldStage)));
        }))
        return XS_CUDA_ERROR;
    const dim3 grid((ls.lines + kFoldLines - 1) / kFoldLines, static_cast<unsigned>(((ls.n + 1) / 2 + kFoldModes - 1) / kFoldModes), batches);
    fold_transform_kernel<kInverse, kStrided, kVec, Tin><<<grid, kFoldThreads, 2 * sizeof(FoldStage), st>>>(in, out, ls, basis);
    return check_launch();
}

template <bool kInverse, bool kStrided, class Tin>
XsStatus transform(cudaStream_t st, const Tin* in, float* out, const FoldLines& ls, uint32_t batches, const float* basis) {
    auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0u; };
    const bool vec = aligned(in) && aligned(out) &&
                     (kStrided ? ls.n % 2 == 0 && ls.stride % 4 == 0 && ls.batch_stride % 4 == 0 && ls.lines % 4 == 0 : ls.n % 8 == 0);
    return vec ? launch_transform<kInverse, kStrided, true, Tin>(st, in, out, ls, batches, basis)
               : launch_transform<kInverse, kStrided, false, Tin>(st, in, out, ls, batches, basis);
}

// ------------------------------------------------------- tridiagonal lines
// (lambda + T) x = b along one axis, in place: lines of `n` values `stride`
// apart, line (i, k) starting at i + k * outer, with lambda = eigen_a[i] +
// eigen_b[k] (transformed axes x and one other).
//
// Elimination from the first value: g_j = w_j (b_j + g_{j-1}), back
// substitution x_j = g_j + w_j x_{j+1}, with w_j the inverse pivots.  Those
// have a closed form: with lambda = 4 sinh(theta / 2)^2 and r = exp(-theta),
//     zero-gradient start: w_j = r (1 + r^(2j+1)) / (1 + r^(2j+3)),
//     fixed start:         w_j = r (1 - r^(2j+2)) / (1 - r^(2j+4)),
// so no division waits for the one before, and a line splits into segments:
// 32 lines (lanes, contiguous in memory) by n / kSeg warps, each keeping a
// segment in registers.  A segment is eliminated from zero, the carries pass
// through shared memory (a carry is multiplied by the product of the w, a
// ratio of the closed form's terms), and the segment is eliminated again with
// the true one; the same backwards.  Small lambda keeps its digits: the last
// pivot, lambda + (1 - w), is evaluated as a product.
constexpr int kSeg = 32;
constexpr int kMaxSegs = kDirectMax / kSeg;

struct TriLines {
    int n;
    uint32_t count_a, count_b;
    uint64_t stride, outer;
    const float *eigen_a, *eigen_b;
    int fixed_lo, fixed_hi;
};

__global__ void __launch_bounds__(kSeg* kMaxSegs) tridiagonal_kernel(float* __restrict__ v, TriLines tl) {
    __shared__ float carry[kMaxSegs][32], factor[kMaxSegs][32];
    const int lane = threadIdx.x, seg = threadIdx.y, segs = blockDim.y;
    const uint32_t ia = blockIdx.x * 32 + lane, ib = blockIdx.y;
    const bool there = ia < tl.count_a;
    const int j0 = seg * kSeg, count = min(kSeg, tl.n - j0);
    float* p = v + (there ? ia : 0u) + static_cast<uint64_t>(ib) * tl.outer + static_cast<uint64_t>(j0) * tl.stride;
    float b[kSeg], w[kSeg];
#pragma unroll
    for (int j = 0; j < kSeg; ++j) b[j] = there && j < count ? p[static_cast<uint64_t>(j) * tl.stride] : 0.0f;
    const float lambda = (there ? __ldg(tl.eigen_a + ia) : 1.0f) + __ldg(tl.eigen_b + ib);
    const float a = 0.5f * sqrtf(lambda), e = 1.0f / (sqrtf(1.0f + a * a) + a);  // sinh(theta / 2), exp(-theta / 2)
    const float r = e * e, one_minus_r = 2.0f * a * e, r2 = r * r;
    const float theta2 = -2.0f * log1pf(-one_minus_r);  // 2 theta
    // zero-gradient: rho_j = r^(2j+1), sign +; fixed: rho_j = r^(2j+2), sign -
    const float sign = tl.fixed_lo ? -1.0f : 1.0f;
    const float first = tl.fixed_lo ? r2 : r;
    float rho = first * expf(-theta2 * static_cast<float>(j0));
    const bool flat = lambda < 1e-30f;  // both transforms' constants: r = 1
    float g = 0.0f, prod = 1.0f, last_w = 0.0f;
#pragma unroll
    for (int j = 0; j < kSeg; ++j) {
        if (flat) {
            const float k = static_cast<float>(j0 + j);
            w[j] = tl.fixed_lo ? (k + 1.0f) / (k + 2.0f) : 1.0f;
        } else if (tl.fixed_lo && (1.0f - rho) < 0.25f) {
            // 1 - r^m for small theta from the exponent
            const float m = 0.5f * theta2 * static_cast<float>(2 * (j0 + j) + 2);
            w[j] = r * expm1f(-m) / expm1f(-m - theta2);
        } else {
            w[j] = r * (1.0f + sign * rho) / (1.0f + sign * rho * r2);
        }
        if (j < count) {
            g = w[j] * (b[j] + g);
            prod *= w[j];
            last_w = w[j];
        }
        rho *= r2;
    }
    carry[seg][lane] = g;
    factor[seg][lane] = prod;
    __syncthreads();
    float in = 0.0f;
    for (int s = 0; s < seg; ++s) in = carry[s][lane] + factor[s][lane] * in;
    __syncthreads();
    // the last pivot belongs to the upper end's row: 2 + lambda - w_{n-2}
    // becomes 1 + lambda - w_{n-2} at a zero-gradient end
    const bool end = j0 + count == tl.n;
    float last_inverse = last_w;
    if (end && !tl.fixed_hi) {
        // 1 / w_{n-1} - 1, as a product where it is small
        float pivot;
        const float jn = static_cast<float>(tl.n - 1);
        if (flat) {
            pivot = tl.fixed_lo ? 1.0f / (jn + 1.0f) : 0.0f;
        } else if (tl.fixed_lo) {
            // 1/w - 1 = (1 - r^(2m+2) - r + r^(2m+1)) / (r (1 - r^2m)), m = n: (1 - r)(1 + r^(2m+1)) / (r (1 - r^2m))
            const float x = 0.5f * theta2;
            pivot = one_minus_r * (1.0f + expf(-x * (2.0f * jn + 3.0f))) / (r * -expm1f(-x * (2.0f * jn + 2.0f)));
        } else {
            // 1/w - 1 = (1 - r)(1 - r^(2n)) / (r (1 + r^(2n-1)))
            const float x = 0.5f * theta2;
            pivot = one_minus_r * -expm1f(-x * (2.0f * jn + 2.0f)) / (r * (1.0f + expf(-x * (2.0f * jn + 1.0f))));
        }
        last_inverse = pivot > 0.0f ? 1.0f / pivot : 0.0f;  // no pivot: the constant of a box without fixed faces
    }
    g = in;
#pragma unroll
    for (int j = 0; j < kSeg; ++j) {
        if (j < count) {
            const float wj = end && j == count - 1 ? last_inverse : w[j];
            g = wj * (b[j] + g);
            b[j] = g;
        }
    }
    // back substitution, segments from the last
    float x = 0.0f;
#pragma unroll
    for (int j = kSeg - 1; j >= 0; --j)
        if (j < count) x = end && j == count - 1 ? b[j] : fmaf(w[j], x, b[j]);
    carry[seg][lane] = x;
    __syncthreads();
    float from = 0.0f;
    for (int s = segs - 1; s > seg; --s) from = carry[s][lane] + (s == segs - 1 ? 0.0f : factor[s][lane] * from);
    x = from;
#pragma unroll
    for (int j = kSeg - 1; j >= 0; --j) {
        if (j < count) {
            x = end && j == count - 1 ? b[j] : fmaf(w[j], x, b[j]);
            if (there) p[static_cast<uint64_t>(j) * tl.stride] = x;
        }
    }
}

bool fold_kind(uint32_t lo, uint32_t hi, int& kind) {
    if (lo == 2u && hi == 2u) { kind = kFoldPeriodic; return true; }
    const bool flo = lo == 0u, fhi = hi == 0u;
    if (flo != fhi) return false;
    kind = flo ? kFoldFixed : kFoldZero;
    return true;
}

}  // namespace

bool direct_plan(const Grid& g, const uint32_t* mask, uint32_t anchor, const XsScalarBoundary& pb, bool fixed_values, DirectPlan& plan) {
    if (mask != nullptr || anchor < cell_count(g) || cell_count(g) >= (1ull << 31)) return false;
    const int n[3] = {g.nx, g.ny, g.nz};
    for (int d = 0; d < 3; ++d)
        if (n[d] < 4 || n[d] > kDirectMax) return false;
    if (fixed_values)
        for (int f = 0; f < 6; ++f)
            if (pb.modes[f] == 0u && pb.values[f] != 0.0f) return false;
    int kind[3];
    bool even[3];
    for (int d = 0; d < 3; ++d) even[d] = fold_kind(pb.modes[2 * d], pb.modes[2 * d + 1], kind[d]);
    if (!even[0]) return false;
    // the tridiagonal axis: y, or z where y is periodic or z has unequal ends
    for (int axis : {1, 2}) {
        const int other = 3 - axis;
        if (!even[other] || (even[axis] && kind[axis] == kFoldPeriodic)) continue;
        plan = DirectPlan{axis, other, kind[0], kind[other], pb.modes[2 * axis] == 0u, pb.modes[2 * axis + 1] == 0u};
        return true;
    }
    return false;
}

size_t direct_basis_bytes() { return sizeof(float) * (2ull * 4 * P * P + 2ull * 2 * P); }

template <class T>
XsStatus direct_solve(cudaStream_t st, const Grid& g, const DirectPlan& plan, const T* rhs, float* tmp, float* tmp2, float* x, void* basis_memory) {
    float* basis = static_cast<float*>(basis_memory);
    float* eigen = basis + 2ull * 4 * P * P;
    const uint64_t nx = g.nx, ny = g.ny, nz = g.nz;
    const int n[3] = {g.nx, g.ny, g.nz};
    const FoldAxes ax{{n[0], n[plan.other]}, {plan.kind_x, plan.kind_other}};
    fold_basis_kernel<<<dim3(P / 32, P / 8, 4), dim3(32, 8), 0, st>>>(ax, basis, eigen);
    XsStatus s = check_launch();
    if (s != XS_OK) return s;
    const FoldLines lx{n[0], static_cast<uint32_t>(ny * nz), 0u, nx, 1u};
    const FoldLines lo = plan.other == 2 ? FoldLines{n[2], static_cast<uint32_t>(nx * ny), 0u, 1u, nx * ny}
                                         : FoldLines{n[1], static_cast<uint32_t>(nx), nx * ny, 1u, nx};
    const uint32_t batches = plan.other == 2 ? 1u : static_cast<uint32_t>(nz);
    const float *bx = basis, *bo = basis + 4ull * P * P;
    if ((s = transform<false, false, T>(st, rhs, tmp, lx, 1u, bx)) != XS_OK) return s;
    if ((s = transform<false, true, float>(st, tmp, tmp2, lo, batches, bo)) != XS_OK) return s;
    const int na = n[plan.axis];
    const TriLines tri{na, static_cast<uint32_t>(nx), static_cast<uint32_t>(n[plan.other]), plan.axis == 1 ? nx : nx * ny,
                       plan.axis == 1 ? nx * ny : nx, eigen, eigen + 2 * P, plan.fixed_lo, plan.fixed_hi};
    tridiagonal_kernel<<<dim3((g.nx + 31) / 32, static_cast<unsigned>(n[plan.other])), dim3(32, (na + kSeg - 1) / kSeg), 0, st>>>(tmp2, tri);
    if ((s = check_launch()) != XS_OK) return s;
    if ((s = transform<true, true, float>(st, tmp2, tmp, lo, batches, bo)) != XS_OK) return s;
    return transform<true, false, float>(st, tmp, x, lx, 1u, bx);
}

template XsStatus direct_solve<float>(cudaStream_t, const Grid&, const DirectPlan&, const float*, float*, float*, float*, void*);
template XsStatus direct_solve<double>(cudaStream_t, const Grid&, const DirectPlan&, const double*, float*, float*, float*, void*);

}  // namespace xs
