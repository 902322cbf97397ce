// 3x3x3 convolutions of the learned pressure warm start on the 5th-generation
// tensor cores (tcgen05), BF16 operands, FP32 accumulation in TMEM.
//
// Activations are NDHWC (channels innermost).  Forward (and the input
// gradient, which is the same convolution with flipped, transposed weights)
// is an implicit GEMM: M = 128 output voxels (a box of the x-y plane at one
// z), N = output channels, K = 27 taps x input channels.  Per tap one TMA
// load brings the shifted 128 x C_in activation box (out-of-range voxels are
// zero-filled by TMA: this is the convolution's zero padding) and one the
// C_out x C_in weight slice, both K-major with the swizzle matching their
// row width; a single thread issues the MMAs; four warps read the
// accumulator back (tcgen05.ld) and apply bias and ReLU.
//
// The weight gradient uses MN-major operands: D[(tap, ci)][co] =
// sum_v X[v + tap][ci] * dY[v][co], M = 128 rows = a group of 128 / C_in taps,
// N = C_out, K = voxels, accumulated in TMEM over a slice of the volume per
// CTA; per-CTA partial sums are reduced in a fixed order by a second kernel.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "launch.cuh"
#include "tc.cuh"
#include "unet.cuh"

namespace xs {

// ------------------------------------------------------------------ TMA maps
namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

CUtensorMapSwizzle swizzle_mode(uint32_t row_bytes) {
    return row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

}  // namespace

// Activation map [B][Z][Y][X][C] with a (C, bx, by, bz, 1) box.
bool make_activation_map(CUtensorMap* map, const void* base, const VolumeShape& s, uint32_t channels, uint32_t bx, uint32_t by, uint32_t bz) {
    auto fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[5] = {channels, s.x, s.y, s.z, s.batch};
    const cuuint64_t e = 2;
    const cuuint64_t strides[4] = {channels * e, s.x * channels * e, static_cast<cuuint64_t>(s.y) * s.x * channels * e,
                                   static_cast<cuuint64_t>(s.z) * s.y * s.x * channels * e};
    const cuuint32_t box[5] = {channels, bx, by, bz, 1};
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              swizzle_mode(channels * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Weight map [27][rows][cols] with a (cols, rows, 1) box: one tap's slice.
bool make_weight_map(CUtensorMap* map, const void* base, uint32_t rows, uint32_t cols) {
    auto fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {cols, rows, 27};
    const cuuint64_t strides[2] = {cols * 2ull, static_cast<cuuint64_t>(rows) * cols * 2ull};
    const cuuint32_t box[3] = {cols, rows, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              swizzle_mode(cols * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ------------------------------------------------------------------ forward
constexpr int kConvThreads = 128;

// Bytes of a CTA's stages: two CTAs per SM, or four.  Deep stages keep the
// MMAs of few CTAs fed, many CTAs do that for one another
// (launch_conv_forward has both sides).
constexpr uint32_t kDeepStages = 98304u, kShallowStages = 49152u;

template <int CIN, int COUT, uint32_t BUDGET>
struct ConvSmem {
    static constexpr uint32_t a_bytes = 128u * CIN * 2u;
    static constexpr uint32_t b_bytes_raw = static_cast<uint32_t>(COUT) * CIN * 2u;
    static constexpr uint32_t b_bytes = (b_bytes_raw + 1023u) / 1024u * 1024u;
    static constexpr uint32_t stage_bytes = a_bytes + b_bytes;
    static constexpr uint32_t fit = BUDGET / stage_bytes;
    static constexpr int stages = fit < 3u ? 3 : (fit < 12u ? static_cast<int>(fit) : 12);
    static constexpr uint32_t total = 1024u /*alignment slack*/ + stages * stage_bytes + 256u /*barriers*/;
    static constexpr uint32_t tmem_cols = COUT <= 32 ? 32u : 64u;
};

struct ConvArgs {
    VolumeShape s;
    uint32_t bx, by, bz;  // output tile box
    const float* bias;
    __nv_bfloat16* out;
    int relu;
    int* error;
};

// One CTA = one tile of 128 output voxels (a bx * by * bz box of one batch).
template <int CIN, int COUT, uint32_t BUDGET>
__global__ void __launch_bounds__(kConvThreads) conv3_forward_kernel(const __grid_constant__ CUtensorMap act_map,
                                                                     const __grid_constant__ CUtensorMap w_map, ConvArgs a) {
    using L = ConvSmem<CIN, COUT, BUDGET>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023u));
    unsigned char* a_tiles = smem;
    unsigned char* b_tiles = smem + L::stages * L::a_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::stages * L::stage_bytes);
    uint64_t* empty = full + L::stages;
    uint64_t* accum = empty + L::stages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);

    const int warp = static_cast<int>(tc::uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;
    // tile coordinates
    const uint32_t tiles_x = a.s.x / a.bx, tiles_y = a.s.y / a.by, tiles_z = a.s.z / a.bz;
    uint32_t t = blockIdx.x;
    const uint32_t tx = t % tiles_x; t /= tiles_x;
    const uint32_t ty = t % tiles_y; t /= tiles_y;
    const uint32_t tz = t % tiles_z;
    const uint32_t b = t / tiles_z;
    const int x0 = static_cast<int>(tx * a.bx), y0 = static_cast<int>(ty * a.by), z0 = static_cast<int>(tz * a.bz);

    if (threadIdx.x == 0) {
        for (int i = 0; i < L::stages; ++i) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 1);
        }
        tc::mbar_init(accum, 1);
        tc::fence_barrier_init();
        tc::prefetch_map(&act_map);
        tc::prefetch_map(&w_map);
    }
    if (warp == 0) {
        tc::tmem_alloc(tmem_slot, L::tmem_cols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tc::uniform(*tmem_slot);
    bool ok = true;

    if (warp == 0) {
        // TMA producer: one stage per tap
        if (tc::elect_one()) {
            for (int tap = 0; tap < 27; ++tap) {
                const int s = tap % L::stages, round = tap / L::stages;
                if (tap >= L::stages && !tc::mbar_wait(&empty[s], (round - 1) & 1)) { ok = false; break; }
                tc::mbar_expect_tx(&full[s], L::a_bytes + L::b_bytes_raw);
                const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
                tc::tma_load_5d(a_tiles + s * L::a_bytes, &act_map, &full[s], 0, x0 + dx, y0 + dy, z0 + dz, static_cast<int>(b));
                tc::tma_load_3d(b_tiles + s * L::b_bytes, &w_map, &full[s], 0, 0, tap);
            }
        }
    } else if (warp == 1) {
        // MMA issuer; the shuffles of uniform() are the whole warp's, before one lane is elected
        constexpr uint32_t idesc = tc::idesc_bf16(128, COUT, false, false);
        constexpr uint32_t row = CIN * 2;
        constexpr uint32_t swz = tc::swizzle_for_row_bytes(row);
        const uint64_t a_desc = tc::smem_desc(tc::uniform(tc::smem_u32(a_tiles)), 16u, 8u * row, swz);
        const uint64_t b_desc = tc::smem_desc(tc::uniform(tc::smem_u32(b_tiles)), 16u, 8u * row, swz);
        if (tc::elect_one()) {
            for (int tap = 0; tap < 27; ++tap) {
                const int s = tap % L::stages, round = tap / L::stages;
                if (!tc::mbar_wait(&full[s], round & 1)) { ok = false; break; }
                tc::tc_fence_after();
                const uint64_t ad = a_desc + (s * L::a_bytes >> 4), bd = b_desc + (s * L::b_bytes >> 4);
#pragma unroll
                for (int k = 0; k < CIN / 16; ++k) tc::mma_bf16(tmem, ad + 2u * k, bd + 2u * k, idesc, (tap > 0 || k > 0) ? 1u : 0u);
                tc::mma_commit(&empty[s]);
            }
            tc::mma_commit(accum);
        }
    }
    __syncwarp();
    // epilogue: every warp reads its 32 TMEM lanes (= voxels)
    const bool got = tc::mbar_wait(accum, 0);
    tc::tc_fence_after();
    if (got) {
        const int r = warp * 32 + lane;
        const int bxy = static_cast<int>(a.bx * a.by);
        const int x = x0 + r % static_cast<int>(a.bx), y = y0 + (r % bxy) / static_cast<int>(a.bx), z = z0 + r / bxy;
        const uint64_t voxel = ((static_cast<uint64_t>(b) * a.s.z + z) * a.s.y + y) * a.s.x + x;
        __nv_bfloat16* dst = a.out + voxel * COUT;
#pragma unroll
        for (int c0 = 0; c0 < COUT; c0 += 16) {
            float v[16];
            tc::tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(c0), v);
            __align__(16) __nv_bfloat16 o[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float y_ = v[i] + (a.bias ? __ldg(a.bias + c0 + i) : 0.0f);
                if (a.relu) y_ = fmaxf(y_, 0.0f);
                o[i] = __float2bfloat16(y_);
            }
            reinterpret_cast<uint4*>(dst + c0)[0] = reinterpret_cast<const uint4*>(o)[0];
            reinterpret_cast<uint4*>(dst + c0)[1] = reinterpret_cast<const uint4*>(o)[1];
        }
    }
    if ((!ok || !got) && a.error) atomicExch(a.error, 1);
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, L::tmem_cols);
}

// ------------------------------------------------------------ halo slab
// The same convolution with the activations read once.  A CTA owns `by` rows
// of `bz` planes and brings their box, widened by one voxel on every side,
// into shared memory: planes of voxels in rows of X + 2, a voxel's channels
// together, 16-byte chunks permuted by their address as the swizzle of that
// row width does.  That is a K-major operand from any voxel on, so a tap is no
// more than another start address: (dy (X + 2) + dx) voxels into plane dz.  A
// tile's 128 rows are consecutive voxels of the widened rows; the two columns
// between rows are computed too and dropped (at X = 64 and 11 rows 92 % of the
// products are kept).  The weights of all 27 taps lie beside it, a barrier each.
//
// What bounds it is the rate at which one warp issues 128 x 16 x 16 MMAs, 40
// cycles each from uniform registers: 16 -> 16 at 64^3 runs in 23.5 us (the
// shifted boxes, 27 x 8.4 MB through L2: 48.6), 8 x 64^3 in 148 (332), of
// which the MMAs are 70.  The unswizzled layout, 8 voxels by 16 bytes at a
// time, gives the same numbers at a quarter of the operand rate: 140 cycles
// per MMA.
constexpr int kSlabThreads = 256;

template <int CIN, int COUT>
struct SlabSmem {
    static constexpr uint32_t chunks = CIN / 8;
    static constexpr uint32_t w_bytes_raw = static_cast<uint32_t>(COUT) * CIN * 2u;
    static constexpr uint32_t w_bytes = (w_bytes_raw + 1023u) / 1024u * 1024u;
    static constexpr uint32_t fixed = 1024u /*alignment*/ + 27u * w_bytes + 512u /*barriers*/;
    static_assert(CIN == 16 && 27u * w_bytes <= 98304u);  // one MMA of K = 16 per tap and tile; room for a box
};
constexpr uint32_t kSlabMaxSmem = 220u * 1024u;
constexpr uint64_t kSlabMinVoxels = 100000u;

struct SlabPlan {
    uint32_t by, bz;      // rows and planes of a CTA
    uint32_t tiles;       // 128-voxel tiles per plane
    uint32_t voxels;      // voxels of a plane's arrays in shared memory
    uint32_t columns;     // TMEM columns
    uint32_t smem;
};

struct SlabArgs {
    VolumeShape s;
    SlabPlan p;
    const __nv_bfloat16* in;
    const float* bias;
    __nv_bfloat16* out;
    int relu;
    int* error;
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kSlabThreads) conv3_slab_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ SlabArgs a) {
    using L = SlabSmem<CIN, COUT>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* taps = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023u));
    uint64_t* full = reinterpret_cast<uint64_t*>(taps + 27u * L::w_bytes);
    uint64_t* accum = full + 27;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    unsigned char* slab = taps + 27u * L::w_bytes + 512;
    const int warp = static_cast<int>(tc::uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;
    const uint32_t strips = (a.s.y + a.p.by - 1) / a.p.by, layers = (a.s.z + a.p.bz - 1) / a.p.bz;
    const uint32_t strip = blockIdx.x % strips, layer = blockIdx.x / strips % layers, b = blockIdx.x / strips / layers;
    const int y0 = static_cast<int>(strip * a.p.by), z0 = static_cast<int>(layer * a.p.bz);
    const int rows = min(static_cast<int>(a.p.by), static_cast<int>(a.s.y) - y0), planes = min(static_cast<int>(a.p.bz), static_cast<int>(a.s.z) - z0);
    const uint32_t px = a.s.x + 2u;
    constexpr uint32_t row_bytes = CIN * 2u;  // of a voxel
    const uint32_t plane_bytes = a.p.voxels * row_bytes;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 27; ++i) tc::mbar_init(&full[i], 1);
        tc::mbar_init(accum, 1);
        tc::fence_barrier_init();
        tc::prefetch_map(&w_map);
    }
    if (warp == 0) {
        tc::tmem_alloc(tmem_slot, a.p.columns);
        tc::tmem_relinquish();
    }
    __syncthreads();
    if (warp == 0 && tc::elect_one()) {
        for (int tap = 0; tap < 27; ++tap) {
            tc::mbar_expect_tx(&full[tap], L::w_bytes_raw);
            tc::tma_load_3d(taps + tap * L::w_bytes, &w_map, &full[tap], 0, 0, tap);
        }
    }
    __syncwarp();
    // the box, zeros beyond the volume: a warp per row, 16 bytes per lane
    for (int r = warp; r < (planes + 2) * (rows + 2); r += kSlabThreads / 32) {
        const int pz = r / (rows + 2), py = r % (rows + 2), z = z0 + pz - 1, y = y0 + py - 1;
        const bool row_in = y >= 0 && y < static_cast<int>(a.s.y) && z >= 0 && z < static_cast<int>(a.s.z);
        const __nv_bfloat16* src = a.in + (((static_cast<uint64_t>(b) * a.s.z + (row_in ? z : 0)) * a.s.y + (row_in ? y : 0)) * a.s.x) * CIN;
        const uint32_t dst = tc::smem_u32(slab) + static_cast<uint32_t>(pz) * plane_bytes + static_cast<uint32_t>(py) * px * row_bytes;
        for (uint32_t j = lane; j < px * L::chunks; j += 32) {
            const uint32_t v = j / L::chunks, c = j % L::chunks;
            const bool in = row_in && v >= 1u && v <= a.s.x;
            const __nv_bfloat16* from = in ? src + (static_cast<uint64_t>(v) - 1u) * CIN + 8u * c : a.in;
            const uint32_t at = dst + v * row_bytes + c * 16u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at ^ (((at >> 7) & (L::chunks - 1u)) << 4)), "l"(from),
                         "r"(in ? 16u : 0u)
                         : "memory");
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the box before the tensor pipe's reads of it
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tc::uniform(*tmem_slot);
    bool ok = true;
    if (warp == 1) {
        constexpr uint32_t idesc = tc::idesc_bf16(128, COUT, false, false);
        // descriptors of the box and of the taps; steps in their 16-byte units
        const uint64_t box = tc::smem_desc(tc::uniform(tc::smem_u32(slab)), 16u, 8u * row_bytes, tc::swizzle_for_row_bytes(row_bytes));
        const uint64_t weights = tc::smem_desc(tc::uniform(tc::smem_u32(taps)), 16u, 8u * row_bytes, tc::swizzle_for_row_bytes(row_bytes));
        constexpr uint32_t tile_step = 128u * row_bytes / 16u;
        const uint32_t plane_step = plane_bytes / 16u, tiles = a.p.tiles;
        if (tc::elect_one()) {
            for (int tap = 0; tap < 27; ++tap) {
                if (!tc::mbar_wait(&full[tap], 0)) { ok = false; break; }
                tc::tc_fence_after();
                const uint32_t dz = static_cast<uint32_t>(tap) / 9u, dy = static_cast<uint32_t>(tap) / 3u % 3u, dx = static_cast<uint32_t>(tap) % 3u;
                const uint64_t w = weights + tap * (L::w_bytes / 16u);
                uint64_t plane = box + dz * plane_step + (dy * px + dx) * (row_bytes / 16u);
                uint32_t d = tmem;
                for (int z = 0; z < planes; ++z) {
                    uint64_t tile = plane;
#pragma unroll 4
                    for (uint32_t t = 0; t < tiles; ++t) {
                        tc::mma_bf16(d, tile, w, idesc, tap > 0 ? 1u : 0u);
                        tile += tile_step;
                        d += COUT;
                    }
                    plane += plane_step;
                }
                // (nothing waits for it: CTAs that share an SM's tensor pipe take
                // turns tap by tap; 16 -> 64 at 128^3 307 us, 327 without)
                tc::mma_commit(&full[tap]);
            }
            tc::mma_commit(accum);
        }
    }
    __syncwarp();
    const bool got = tc::mbar_wait(accum, 0);
    tc::tc_fence_after();
    if (got) {
        // warps 0-3 take the even tiles, 4-7 the odd ones, 32 rows each
        for (uint32_t i = static_cast<uint32_t>(warp >> 2); i < static_cast<uint32_t>(planes) * a.p.tiles; i += 2u) {
            const uint32_t pz = i / a.p.tiles, t = i - pz * a.p.tiles;
            const uint32_t v = t * 128u + static_cast<uint32_t>((warp & 3) * 32 + lane), r = v / px, x = v - r * px;
            const bool keep = x < a.s.x && r < static_cast<uint32_t>(rows);
            const uint64_t voxel = ((static_cast<uint64_t>(b) * a.s.z + static_cast<uint32_t>(z0) + pz) * a.s.y + static_cast<uint32_t>(y0) + r) * a.s.x + x;
            __nv_bfloat16* dst = a.out + voxel * COUT;
#pragma unroll
            for (int c0 = 0; c0 < COUT; c0 += 16) {
                float f[16];
                tc::tmem_ld16(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + i * COUT + static_cast<uint32_t>(c0), f);
                __align__(16) __nv_bfloat16 o[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    float y_ = f[e] + (a.bias ? __ldg(a.bias + c0 + e) : 0.0f);
                    if (a.relu) y_ = fmaxf(y_, 0.0f);
                    o[e] = __float2bfloat16(y_);
                }
                if (keep) {
                    reinterpret_cast<uint4*>(dst + c0)[0] = reinterpret_cast<const uint4*>(o)[0];
                    reinterpret_cast<uint4*>(dst + c0)[1] = reinterpret_cast<const uint4*>(o)[1];
                }
            }
        }
    }
    if ((!ok || !got) && a.error) atomicExch(a.error, 1);
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, a.p.columns);
}

// The rows and planes of a CTA that take the least time on 148 SMs, from a fit
// to 174 strips of 16 -> 16 at 64^3, 8 x 64^3, 128^3 and 128 x 128 x 64: a wave
// of r CTAs per SM (by shared memory and TMEM) costs 10 us for the box, the
// launch and the epilogue, and per MMA of a CTA 20 ns and 11 ns more for each of
// the r that share the tensor pipe.  Its picks took 23.0, 152.7, 158.1 and
// 89.6 us; the best strips 23.0, 143.0, 158.1 and 89.6.  (Counting the parts of
// one CTA in cycles picked 26.9, 158.5, 158.2 and 98.6.)  The constants serve
// 16 -> 32 and 16 -> 64 unfitted, whose MMAs take longer: against the boxes 64^3
// 30.4 (50.8) and 50.8 (65.6), 128^3 219 (344) and 308 (463), 8 x 64^3 162 (345)
// and 345 (463).  Of 13 shapes of 131,072 voxels and more the boxes are faster in
// one, 16 -> 64 at 8 x 16 x 1024 (37.3 against 39.1): rows of 8 in rows of 10.
template <int CIN, int COUT>
bool slab_plan(const VolumeShape& s, SlabPlan& best) {
    using L = SlabSmem<CIN, COUT>;
    double least = 0.0;
    const uint32_t px = s.x + 2u;
    for (uint32_t bz = 1; bz <= std::min(4u, s.z); ++bz)
        for (uint32_t by = 1; by <= s.y; ++by) {
            SlabPlan p{};
            p.by = by;
            p.bz = bz;
            p.tiles = ((by - 1) * px + s.x + 127u) / 128u;
            p.voxels = std::max((by + 2) * px, p.tiles * 128u + 2u * px + 2u);
            p.columns = 32u;
            while (p.columns < bz * p.tiles * COUT) p.columns *= 2;
            const uint64_t smem = L::fixed + static_cast<uint64_t>(bz + 2) * p.voxels * CIN * 2u;
            if (p.columns > 512u || smem > kSlabMaxSmem) break;
            p.smem = static_cast<uint32_t>(smem);
            const uint64_t ctas = static_cast<uint64_t>(s.batch) * ((s.z + bz - 1) / bz) * ((s.y + by - 1) / by);
            const uint64_t resident = std::min({227ull * 1024u / (smem + 1024u), 512ull / p.columns, (ctas + 147ull) / 148u});
            const double waves = static_cast<double>((ctas + 148u * resident - 1u) / (148u * resident));
            const double cost = 10.0 + 27.0 * (bz * p.tiles * (CIN / 16)) * (0.020 + 0.011 * static_cast<double>(resident));
            if (least == 0.0 || waves * cost < least) {
                least = waves * cost;
                best = p;
            }
        }
    return least > 0.0;
}

template <int CIN, int COUT>
XsStatus launch_conv_slab(cudaStream_t st, const VolumeShape& s, const SlabPlan& plan, const __nv_bfloat16* in, const __nv_bfloat16* w, const float* bias,
                          __nv_bfloat16* out, bool relu, int* error) {
    CUtensorMap wm;
    // (the box copies are of 16 bytes, as a tensor map's base has to be)
    if ((reinterpret_cast<uintptr_t>(in) & 15u) || !make_weight_map(&wm, w, COUT, CIN)) return XS_CUDA_ERROR;
    static DeviceOnce configured;
    if (!configured.run([] { return cudaFuncSetAttribute(conv3_slab_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSlabMaxSmem)); }))
        return XS_CUDA_ERROR;
    const SlabArgs args{s, plan, in, bias, out, relu ? 1 : 0, error};
    const uint64_t ctas = static_cast<uint64_t>(s.batch) * ((s.z + plan.bz - 1) / plan.bz) * ((s.y + plan.by - 1) / plan.by);
    conv3_slab_kernel<CIN, COUT><<<static_cast<unsigned>(ctas), kSlabThreads, plan.smem, st>>>(wm, args);
    return check_launch();
}

template <int CIN, int COUT, uint32_t BUDGET>
XsStatus launch_conv_boxes(cudaStream_t st, const CUtensorMap& am, const CUtensorMap& wm, const ConvArgs& args, uint64_t tiles) {
    using L = ConvSmem<CIN, COUT, BUDGET>;
    static DeviceOnce configured;
    if (!configured.run([] { return cudaFuncSetAttribute(conv3_forward_kernel<CIN, COUT, BUDGET>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::total); }))
        return XS_CUDA_ERROR;
    conv3_forward_kernel<CIN, COUT, BUDGET><<<static_cast<unsigned>(tiles), kConvThreads, L::total, st>>>(am, wm, args);
    return check_launch();
}

template <int CIN, int COUT>
XsStatus launch_conv_forward(cudaStream_t st, const VolumeShape& s, const __nv_bfloat16* in, const __nv_bfloat16* w, const float* bias,
                             __nv_bfloat16* out, bool relu, int* error) {
    uint32_t bx, by, bz;
    if (!conv_tile(s, bx, by, bz)) return XS_INVALID_ARGUMENT;
    // The slab wins where the 27 shifted boxes of narrow layers fill the SMs:
    // 16 -> 16 at 64^3 23.5 us against 48.6 from the boxes, at 8 x 64^3 148
    // against 332; 16 -> 32 at 8 x 32^3 29 against 50.  With fewer voxels a CTA
    // has too few MMAs behind one box to wait for (16 -> 32 at 32^3 14.1 us
    // against 11.1; by both slopes they meet near 100,000 voxels), and from 32
    // channels on a box fills an MMA's time anyway (32 -> 16 at 8 x 32^3 52.0
    // against 39.1, 64 -> 64 at 16^3 16.2 against 9.9).
    if constexpr (CIN == 16) {
        SlabPlan plan;
        if (static_cast<uint64_t>(s.x) * s.y * s.z * s.batch >= kSlabMinVoxels && slab_plan<CIN, COUT>(s, plan))
            return launch_conv_slab<CIN, COUT>(st, s, plan, in, w, bias, out, relu, error);
    }
    CUtensorMap am, wm;
    if (!make_activation_map(&am, in, s, CIN, bx, by, bz) || !make_weight_map(&wm, w, COUT, CIN)) return XS_CUDA_ERROR;
    const ConvArgs args{s, bx, by, bz, bias, out, relu ? 1 : 0, error};
    const uint64_t tiles = static_cast<uint64_t>(s.batch) * (s.z / bz) * (s.y / by) * (s.x / bx);
    // Few tiles: deep stages, 64 -> 64 with 128 tiles 10.5 us (shallow 12.5), 16 ->
    // 64 with 512 22.9 (27.0).  Many: shallow ones and twice the CTAs, with 2,048
    // tiles 32 -> 16 39.1 (deep 51.2), 32 -> 32 47.4 (55.5), 64 -> 16 56.3 (63.4), 64
    // -> 64 76.3 (78.2), with 12,284 32 -> 16 196 (277).  They meet between 512 and
    // 1,024 tiles; before that where a tile's products are few, 32 channels to at
    // most 32 (456 tiles, 32 -> 16 14.5, deep 16.5; 32 -> 32 17.3, deep 18.6), and
    // where its box is many short rows, x of 2 or 4 (340 to 426 tiles, 64 -> 32 14.6
    // to 16.5, deep 16.7 to 18.7; 160, 64 -> 32 12.4, deep 10.6).
    const bool early = (CIN == 32 && COUT <= 32) || s.x < 8u;
    const uint64_t few = 148u * (early ? 2u : 4u);
    return tiles <= few ? launch_conv_boxes<CIN, COUT, kDeepStages>(st, am, wm, args, tiles)
                        : launch_conv_boxes<CIN, COUT, kShallowStages>(st, am, wm, args, tiles);
}

// The 128-voxel output tile: as wide in x as the volume allows (up to 128),
// then in y, then in z (for small volumes, several z planes per tile).
bool conv_tile(const VolumeShape& s, uint32_t& bx, uint32_t& by, uint32_t& bz) {
    bx = s.x < 128 ? s.x : 128;
    if (bx == 0 || 128 % bx != 0 || s.x % bx != 0) return false;
    by = 128 / bx < s.y ? 128 / bx : s.y;
    if (by == 0 || (128 / bx) % by != 0 || s.y % by != 0) return false;
    bz = 128 / (bx * by);
    return bz <= s.z && s.z % bz == 0;
}

XsStatus conv3_forward(cudaStream_t st, const VolumeShape& s, int cin, int cout, const __nv_bfloat16* in, const __nv_bfloat16* w,
                       const float* bias, __nv_bfloat16* out, bool relu, int* error) {
#define XS_CONV_CASE(CI, CO) \
    if (cin == CI && cout == CO) return launch_conv_forward<CI, CO>(st, s, in, w, bias, out, relu, error);
    XS_CONV_CASE(16, 16) XS_CONV_CASE(16, 32) XS_CONV_CASE(16, 64)
    XS_CONV_CASE(32, 16) XS_CONV_CASE(32, 32) XS_CONV_CASE(32, 64)
    XS_CONV_CASE(64, 16) XS_CONV_CASE(64, 32) XS_CONV_CASE(64, 64)
#undef XS_CONV_CASE
    return XS_INVALID_ARGUMENT;
}

// ------------------------------------------------------------------ weight gradient
// D[(tap, ci)][co] = sum over voxels v of X[v + tap][ci] * dY[v][co].
// Rows: a group of G = 128 / C_in taps (the G shifted activation boxes sit
// in consecutive tiles, one MN-major atom each); columns: C_out; K: the 128
// voxels of a tile.  A CTA owns a slice of the voxel tiles and a set of tap
// groups whose accumulators fit 256 TMEM columns.
template <int CIN, int COUT>
struct WgradLayout {
    static constexpr int G = 128 / CIN;
    static constexpr int groups = (27 + G - 1) / G;
    static constexpr int groups_per_set = 256 / COUT;
    static constexpr int sets = (groups + groups_per_set - 1) / groups_per_set;
    static constexpr uint32_t x_tile = 128u * CIN * 2u;
    static constexpr uint32_t y_bytes = 128u * COUT * 2u;
    static constexpr uint32_t y_padded = (y_bytes + 1023u) / 1024u * 1024u;
    static constexpr uint32_t stage_bytes = G * x_tile + y_padded;
    static constexpr int stages = 3;
    static constexpr uint32_t total = 1024u + stages * stage_bytes + 256u;
};

constexpr uint32_t kWgradCtas = 148u;  // most CTAs of a weight gradient, one per SM

struct WgradArgs {
    VolumeShape s;
    uint32_t bx, by, bz;
    uint32_t tiles;
    float* partial;  // [gridDim.x][27][COUT][CIN]
    int* error;
    // After slabs: their CTAs' flags and a ticket.  Without a flag set their sums
    // are added up here; with one the sums are formed again, and added up by
    // the last CTA to finish.
    const uint32_t* redo;  // null: not after slabs
    uint32_t redo_count;
    uint32_t* ticket;
    float* dw;
    int accumulate;
};

// dW[i] (+)= sum over CTAs of partial[cta][i], in CTA order, for i = first,
// first + step, ... (kSums of them), with 32 loads of each in flight.
template <int kSums>
struct PartialSums {
    float acc[kSums];
    __device__ __forceinline__ void form(const float* partial, uint32_t ctas, uint32_t count, uint32_t first, uint32_t step) {
#pragma unroll
        for (int k = 0; k < kSums; ++k) acc[k] = 0.0f;
        for (uint32_t c0 = 0; c0 < ctas; c0 += 32u) {
            float v[kSums][32];
#pragma unroll
            for (int k = 0; k < kSums; ++k)
#pragma unroll
                for (uint32_t c = 0; c < 32u; ++c)
                    if (c0 + c < ctas && first + k * step < count) v[k][c] = __ldcg(partial + static_cast<size_t>(c0 + c) * count + first + k * step);
#pragma unroll
            for (int k = 0; k < kSums; ++k)
#pragma unroll
                for (uint32_t c = 0; c < 32u; ++c)
                    if (c0 + c < ctas && first + k * step < count) acc[k] += v[k][c];
        }
    }
    __device__ __forceinline__ void add_to(float* dw, int accumulate, uint32_t count, uint32_t first, uint32_t step) const {
#pragma unroll
        for (int k = 0; k < kSums; ++k) {
            const uint32_t i = first + k * step;
            if (i < count) dw[i] = accumulate ? dw[i] + acc[k] : acc[k];
        }
    }
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kConvThreads) conv3_wgrad_kernel(const __grid_constant__ CUtensorMap x_map,
                                                                   const __grid_constant__ CUtensorMap dy_map, WgradArgs a) {
    constexpr uint32_t count = 27u * CIN * COUT;
    constexpr bool kAfterSlabs = CIN <= 32 && COUT <= 32;
    if constexpr (kAfterSlabs) if (a.redo) {
        // the sums are formed while the flags are on their way; a CTA per SM
        // (more do not fit beside the boxes' memory)
        constexpr int kSums = (count + kWgradCtas * kConvThreads - 1u) / (kWgradCtas * kConvThreads);
        const uint32_t first = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x, step = gridDim.x * gridDim.y * blockDim.x;
        bool any = false;
        for (uint32_t i = threadIdx.x; i < a.redo_count; i += blockDim.x) any |= __ldcg(a.redo + i) != 0u;
        PartialSums<kSums> sums;
        sums.form(a.partial, a.redo_count, count, first, step);
        if (!__syncthreads_or(any)) {
            sums.add_to(a.dw, a.accumulate, count, first, step);
            for (uint32_t i = first + kSums * step; i < count; i += kSums * step) {
                sums.form(a.partial, a.redo_count, count, i, step);
                sums.add_to(a.dw, a.accumulate, count, i, step);
            }
            return;
        }
    }
    using L = WgradLayout<CIN, COUT>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023u));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::stages * L::stage_bytes);
    uint64_t* empty = full + L::stages;
    uint64_t* accum = empty + L::stages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    const int warp = static_cast<int>(tc::uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;

    const uint32_t cx = blockIdx.x, nctas = gridDim.x;
    const uint32_t t_begin = static_cast<uint32_t>(static_cast<uint64_t>(a.tiles) * cx / nctas);
    const uint32_t t_end = static_cast<uint32_t>(static_cast<uint64_t>(a.tiles) * (cx + 1) / nctas);
    const int g_begin = static_cast<int>(blockIdx.y) * L::groups_per_set;
    const int g_count = min(L::groups_per_set, L::groups - g_begin);
    const uint32_t items = (t_end - t_begin) * static_cast<uint32_t>(g_count);

    if (threadIdx.x == 0) {
        for (int i = 0; i < L::stages; ++i) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 1);
        }
        tc::mbar_init(accum, 1);
        tc::fence_barrier_init();
        tc::prefetch_map(&x_map);
        tc::prefetch_map(&dy_map);
    }
    if (warp == 0) {
        tc::tmem_alloc(tmem_slot, 256);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tc::uniform(*tmem_slot);
    bool ok = true;
    const uint32_t tiles_x = a.s.x / a.bx, tiles_y = a.s.y / a.by, tiles_z = a.s.z / a.bz;

    if (warp == 0) {
      if (tc::elect_one()) {
        for (uint32_t i = 0; i < items; ++i) {
            const int s = static_cast<int>(i % L::stages), round = static_cast<int>(i / L::stages);
            if (i >= static_cast<uint32_t>(L::stages) && !tc::mbar_wait(&empty[s], (round - 1) & 1)) { ok = false; break; }
            const uint32_t tile = t_begin + i / g_count;
            const int group = g_begin + static_cast<int>(i % g_count);
            uint32_t t = tile;
            const uint32_t tx = t % tiles_x; t /= tiles_x;
            const uint32_t ty = t % tiles_y; t /= tiles_y;
            const int z = static_cast<int>((t % tiles_z) * a.bz), b = static_cast<int>(t / tiles_z);
            const int x0 = static_cast<int>(tx * a.bx), y0 = static_cast<int>(ty * a.by);
            unsigned char* st = smem + s * L::stage_bytes;
            tc::mbar_expect_tx(&full[s], L::G * L::x_tile + L::y_bytes);
            for (int j = 0; j < L::G; ++j) {
                const int tap = group * L::G + j;
                if (tap < 27) {
                    const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
                    tc::tma_load_5d(st + j * L::x_tile, &x_map, &full[s], 0, x0 + dx, y0 + dy, z + dz, b);
                } else {  // missing taps of the last group: a box far outside the volume reads zeros
                    tc::tma_load_5d(st + j * L::x_tile, &x_map, &full[s], 0, 0, 0, -static_cast<int>(2 * a.bz + 64), 0);
                }
            }
            tc::tma_load_5d(st + L::G * L::x_tile, &dy_map, &full[s], 0, x0, y0, z, b);
        }
      }
    } else if (warp == 1) {
        constexpr uint32_t idesc = tc::idesc_bf16(128, COUT, true, true);
        constexpr uint32_t a_row = CIN * 2, b_row = COUT * 2;
        const uint32_t first = tc::uniform(tc::smem_u32(smem));
        const uint64_t xs_desc = tc::smem_desc(first, L::x_tile, 8u * a_row, tc::swizzle_for_row_bytes(a_row));
        const uint64_t dy_desc = tc::smem_desc(first + L::G * L::x_tile, L::y_padded, 8u * b_row, tc::swizzle_for_row_bytes(b_row));
        if (tc::elect_one()) {
            uint32_t s = 0u, round = 0u, group = 0u, accumulate = 0u;
            for (uint32_t i = 0; i < items; ++i) {
                if (!tc::mbar_wait(&full[s], round & 1u)) { ok = false; break; }
                tc::tc_fence_after();
                const uint64_t xd = xs_desc + s * (L::stage_bytes / 16u), yd = dy_desc + s * (L::stage_bytes / 16u);
                const uint32_t d = tmem + group * COUT;
#pragma unroll
                for (uint32_t k = 0; k < 8u; ++k)  // 16 voxels per MMA: two 8-row atoms
                    tc::mma_bf16(d, xd + k * a_row, yd + k * b_row, idesc, k > 0u ? 1u : accumulate);
                tc::mma_commit(&empty[s]);
                if (++s == static_cast<uint32_t>(L::stages)) { s = 0u; ++round; }
                if (++group == static_cast<uint32_t>(g_count)) { group = 0u; accumulate = 1u; }
            }
            tc::mma_commit(accum);
        }
    }
    __syncwarp();
    const bool got = items == 0 ? true : tc::mbar_wait(accum, 0);
    tc::tc_fence_after();
    if (got && items > 0) {
        const int m = warp * 32 + lane;
        const int j = m / CIN, ci = m % CIN;
        for (int gl = 0; gl < g_count; ++gl) {
            const int tap = (g_begin + gl) * L::G + j;
#pragma unroll
            for (int c0 = 0; c0 < COUT; c0 += 16) {
                float v[16];
                tc::tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(gl * COUT + c0), v);
                if (tap < 27) {
                    float* dst = a.partial + ((static_cast<size_t>(cx) * 27 + tap) * COUT + c0) * CIN + ci;
#pragma unroll
                    for (int q = 0; q < 16; ++q) dst[static_cast<size_t>(q) * CIN] = v[q];
                }
            }
        }
    }
    if ((!ok || !got) && a.error) atomicExch(a.error, 1);
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 256);
    if constexpr (kAfterSlabs) {
        if (!a.redo) return;
        __shared__ uint32_t before;
        __threadfence();  // the CTA's sums before its ticket
        __syncthreads();
        if (threadIdx.x == 0) before = atomicAdd(a.ticket, 1u);
        __syncthreads();
        if (before != gridDim.x * gridDim.y - 1u) return;
        __threadfence();
        PartialSums<1> sums;
        for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
            sums.form(a.partial, nctas, count, i, 0u);
            sums.add_to(a.dw, a.accumulate, count, i, 0u);
        }
    }
}

// -------------------------------------------- weight gradient, read once
// The same sums for up to 32 channels on either side, with every voxel brought
// into shared memory once instead of once per tap.  A CTA walks the planes of
// a strip of R rows; its planes of X are kept in rows of X + 1 voxels behind
// a column of zeros, R of them, those of dY the same way with a row more on
// either side, three deep.  In these rows two voxels that a tap pairs are the
// same distance apart everywhere, and a pair that wraps around a row's end has
// a zero in it, so 16 consecutive voxels of X and of dY are one K step for all
// taps at once: the rows of the MMA are X from 128 / C_in consecutive
// voxels on (its operand's atoms overlap, one voxel apart; the first three are
// the taps' dx), the columns dY from three consecutive rows on (dy), one MMA
// and one accumulator per plane of dY (dz).
//
// What bounds it is one warp's MMA issue, 3 per 16 voxels; the boxes per tap
// are bound by L2 instead (27 x 67 MB at 8 x 64^3).16 -> 16 at
// 8 x 64^3: 82.8 us (298), where the MMAs, 128 x 48 x 16 at 45 cycles, are 65.
//
// A voxel that is infinite or NaN also meets zeros here that no tap pairs it
// with (a row's margin), which turn taps NaN that it is not in.  A CTA whose
// sums are not all finite raises its flag, and the kernel that would add up the
// CTAs' sums then forms them again from boxes.
constexpr uint64_t kWslabMinVoxels = 30000u;
constexpr uint32_t kWsTail = 32u;  // voxels of zeros past a plane: a K step's rest and the atoms' shifts

struct WslabArgs {
    VolumeShape s;
    uint32_t rows;      // R
    uint32_t strips;    // per plane
    uint32_t slots;     // planes in flight
    uint32_t x_bytes, slot_bytes;
    float* partial;     // [gridDim.x][27][COUT][CIN]
    uint32_t* redo;     // [gridDim.x]: 1 where a sum is not finite
    uint32_t* ticket;   // of what follows, cleared here
    int* error;
};
constexpr uint32_t kWsMaxSlots = 8u;

template <int CIN, int COUT>
__global__ void __launch_bounds__(kConvThreads) conv3_wgrad_slab_kernel(const __grid_constant__ CUtensorMap x_map,
                                                                        const __grid_constant__ CUtensorMap dy_map, WslabArgs a) {
    constexpr uint32_t x_voxel = CIN * 2u, y_voxel = COUT * 2u, columns = 9u * COUT <= 256u ? 256u : 512u;
    static_assert(128 / CIN >= 3 && 9 * COUT <= 512);
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023u));
    __shared__ uint64_t full[kWsMaxSlots], empty[kWsMaxSlots], accum[1];
    __shared__ uint32_t tmem_slot;
    const int warp = static_cast<int>(tc::uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;
    const uint32_t px = a.s.x + 1u, x_box = a.rows * px * x_voxel, y_box = (a.rows + 2u) * px * y_voxel;
    const uint64_t items = static_cast<uint64_t>(a.s.batch) * a.strips * a.s.z;
    const uint32_t first = static_cast<uint32_t>(items * blockIdx.x / gridDim.x), last = static_cast<uint32_t>(items * (blockIdx.x + 1u) / gridDim.x);

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < a.slots; ++i) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 1);
        }
        tc::mbar_init(accum, 1);
        tc::fence_barrier_init();
        tc::prefetch_map(&x_map);
        tc::prefetch_map(&dy_map);
    }
    if (warp == 0) {
        tc::tmem_alloc(&tmem_slot, columns);
        tc::tmem_relinquish();
    }
    for (uint32_t i = threadIdx.x; i < a.slots * kWsTail * (x_voxel + y_voxel) / 4u; i += kConvThreads) {
        const uint32_t slot = i / (kWsTail * (x_voxel + y_voxel) / 4u), w = i % (kWsTail * (x_voxel + y_voxel) / 4u), xw = kWsTail * x_voxel / 4u;
        unsigned char* at = smem + slot * a.slot_bytes + (w < xw ? x_box + w * 4u : a.x_bytes + y_box + (w - xw) * 4u);
        *reinterpret_cast<uint32_t*>(at) = 0u;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tc::uniform(tmem_slot);
    bool ok = true;

    // Both sides walk the same stages: for the planes [z, z + n) of a strip
    // that this CTA owns, the planes [z - 1, z + n] of dY, and from the third
    // stage on a plane of X two behind, for which the three are there.  Stage
    // g gives back the slot of stage g - 2.
    if (warp == 0) {
        if (tc::elect_one()) {
            uint32_t slot = 0u, round = 0u;
            for (uint32_t i = first; i < last && ok;) {
                const uint32_t z = i % a.s.z, column = i / a.s.z, n = min(a.s.z - z, last - i);
                const int y0 = static_cast<int>(column % a.strips * a.rows), b = static_cast<int>(column / a.strips);
                for (uint32_t t = 0; t < n + 2u; ++t) {
                    if (round > 0u && !tc::mbar_wait(&empty[slot], (round - 1u) & 1u)) { ok = false; break; }
                    unsigned char* at = smem + slot * a.slot_bytes;
                    tc::mbar_expect_tx(&full[slot], y_box + (t >= 2u ? x_box : 0u));
                    tc::tma_load_5d(at + a.x_bytes, &dy_map, &full[slot], 0, -1, y0 - 1, static_cast<int>(z + t) - 1, b);
                    if (t >= 2u) tc::tma_load_5d(at, &x_map, &full[slot], 0, -1, y0, static_cast<int>(z + t) - 2, b);
                    if (++slot == a.slots) { slot = 0u; ++round; }
                }
                i += n;
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = tc::idesc_bf16(128, 3 * COUT, true, true);
        const uint32_t at = tc::uniform(tc::smem_u32(smem));
        // atoms one voxel apart (X) and one row apart (dY, which starts a voxel on)
        const uint64_t x_desc = tc::smem_desc(at, x_voxel, 8u * x_voxel, tc::swizzle_for_row_bytes(x_voxel));
        const uint64_t y_desc = tc::smem_desc(at + a.x_bytes + y_voxel, px * y_voxel, 8u * y_voxel, tc::swizzle_for_row_bytes(y_voxel));
        const uint32_t step = a.slot_bytes / 16u;
        if (tc::elect_one()) {
            uint32_t slot = 0u, round = 0u, before = 0u, two_before = 0u, accumulate = 0u, stages = 0u;
            for (uint32_t i = first; i < last && ok;) {
                const uint32_t z = i % a.s.z, column = i / a.s.z, n = min(a.s.z - z, last - i);
                const uint32_t steps = (min(a.rows, a.s.y - column % a.strips * a.rows) * px + 15u) / 16u;
                for (uint32_t t = 0; t < n + 2u; ++t, ++stages) {
                    if (!tc::mbar_wait(&full[slot], round & 1u)) { ok = false; break; }
                    if (t >= 2u) {
                        tc::tc_fence_after();
                        uint64_t xd = x_desc + slot * step, y0 = y_desc + two_before * step, y1 = y_desc + before * step, y2 = y_desc + slot * step;
#pragma unroll 2
                        for (uint32_t k = 0; k < steps; ++k) {
                            tc::mma_bf16(tmem, xd, y0, idesc, accumulate);
                            tc::mma_bf16(tmem + 3u * COUT, xd, y1, idesc, accumulate);
                            tc::mma_bf16(tmem + 6u * COUT, xd, y2, idesc, accumulate);
                            xd += x_voxel;  // 16 voxels, in units of 16 bytes
                            y0 += y_voxel;
                            y1 += y_voxel;
                            y2 += y_voxel;
                            accumulate = 1u;
                        }
                    }
                    if (stages >= 2u) tc::mma_commit(&empty[two_before]);
                    two_before = before;
                    before = slot;
                    if (++slot == a.slots) { slot = 0u; ++round; }
                }
                i += n;
            }
            tc::mma_commit(accum);
        }
    }
    __syncwarp();
    const bool got = tc::mbar_wait(accum, 0);
    tc::tc_fence_after();
    bool finite = true;
    if (got && warp * 32 < 3 * CIN) {
        const int m = warp * 32 + lane, dx = m / CIN, ci = m % CIN;
        for (int d = 0; d < 9; ++d) {  // planes of dY in rising order fall to taps of falling dz, rows to dy
            const int tap = (2 - d / 3) * 9 + (2 - d % 3) * 3 + dx;
#pragma unroll
            for (int c0 = 0; c0 < COUT; c0 += 16) {
                float v[16];
                tc::tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(d * COUT + c0), v);
                if (dx < 3) {
                    float* dst = a.partial + ((static_cast<size_t>(blockIdx.x) * 27 + tap) * COUT + c0) * CIN + ci;
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        dst[static_cast<size_t>(q) * CIN] = v[q];
                        finite &= isfinite(v[q]);
                    }
                }
            }
        }
    }
    if ((!ok || !got) && a.error) atomicExch(a.error, 1);
    tc::tc_fence_before();
    const bool again = __syncthreads_or(!finite) != 0;
    if (threadIdx.x == 0) {
        a.redo[blockIdx.x] = again ? 1u : 0u;
        if (blockIdx.x == 0) *a.ticket = 0u;
    }
    if (warp == 0) tc::tmem_dealloc(tmem, columns);
}

// Rows of a strip: the fewest MMAs on the CTA with the most of them, with room
// for a plane in flight beside the three in use.
template <int CIN, int COUT>
bool wgrad_slab_plan(const VolumeShape& s, uint32_t ctas, WslabArgs& best) {
    const uint32_t px = s.x + 1u;
    if (px > 256u) return false;  // the widest box of a tensor map
    uint64_t least = 0u;
    for (uint32_t rows = 1; rows <= std::min(s.y, 254u); ++rows) {
        const uint32_t x_bytes = ((rows * px + kWsTail) * CIN * 2u + 1023u) / 1024u * 1024u;
        const uint32_t slot = x_bytes + (((rows + 2u) * px + kWsTail) * COUT * 2u + 1023u) / 1024u * 1024u;
        const uint32_t slots = std::min(kWsMaxSlots, (kSlabMaxSmem - 1024u) / slot);
        if (slots < 4u) break;
        const uint32_t strips = (s.y + rows - 1u) / rows;
        const uint64_t items = static_cast<uint64_t>(s.batch) * strips * s.z, of_one = (items + ctas - 1u) / ctas;
        // 45 cycles an MMA, a stage's hand-over, and two planes more where a strip begins
        const uint64_t cycles = of_one * (3u * ((rows * px + 15u) / 16u) * 45u + 200u) + 2u * (of_one / s.z + 1u) * 400u;
        if (least == 0u || cycles < least) {
            least = cycles;
            best = WslabArgs{s, rows, strips, slots, x_bytes, slot, nullptr, nullptr, nullptr, nullptr};
        }
    }
    return least > 0u;
}

// dW (+)= the sums over CTAs of their parts.
__global__ void wgrad_reduce_kernel(const float* __restrict__ partial, uint32_t ctas, uint32_t count, float* __restrict__ dw, int accumulate) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float acc = 0.0f;
    for (uint32_t c = 0; c < ctas; ++c) acc += partial[static_cast<size_t>(c) * count + i];
    dw[i] = accumulate ? dw[i] + acc : acc;
}

uint32_t wgrad_ctas(const VolumeShape& s) {
    uint32_t bx, by, bz;
    if (!conv_tile(s, bx, by, bz)) return 0;
    const uint64_t tiles = static_cast<uint64_t>(s.batch) * (s.z / bz) * (s.y / by) * (s.x / bx);
    return static_cast<uint32_t>(tiles < kWgradCtas ? tiles : kWgradCtas);
}

// (the partial sums, and behind them a flag per CTA and a ticket)
size_t wgrad_partial_floats(const VolumeShape& s, int cin, int cout) {
    const size_t ctas = wgrad_ctas(s);
    return ctas == 0 ? 0 : ctas * (27u * static_cast<size_t>(cin) * static_cast<size_t>(cout) + 1u) + 1u;
}

template <int CIN, int COUT>
XsStatus launch_wgrad(cudaStream_t st, const VolumeShape& s, const __nv_bfloat16* x, const __nv_bfloat16* dy, float* partial, float* dw,
                      bool accumulate, int* error) {
    using L = WgradLayout<CIN, COUT>;
    uint32_t bx, by, bz;
    if (!conv_tile(s, bx, by, bz)) return XS_INVALID_ARGUMENT;
    CUtensorMap xm, ym;
    if (!make_activation_map(&xm, x, s, CIN, bx, by, bz) || !make_activation_map(&ym, dy, s, COUT, bx, by, bz)) return XS_CUDA_ERROR;
    static DeviceOnce configured;
    if (!configured.run([] { return cudaFuncSetAttribute(conv3_wgrad_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::total); }))
        return XS_CUDA_ERROR;
    const uint32_t tiles = static_cast<uint32_t>(static_cast<uint64_t>(s.batch) * (s.z / bz) * (s.y / by) * (s.x / bx));
    const uint32_t ctas = wgrad_ctas(s);
    const uint32_t count = 27u * CIN * COUT;
    WgradArgs args{s, bx, by, bz, tiles, partial, error, nullptr, 0u, nullptr, dw, accumulate ? 1 : 0};
    if constexpr (CIN <= 32 && COUT <= 32) {
        // 16 -> 16 at 8 x 64^3 82.8 us against 298 from the boxes, at 64^3 22.9
        // against 48.0, at 32^3 14.5 against 16.5, where a CTA has 6 planes
        // and two thirds of the time is the launches and the wait for its
        // first three loads; 32 -> 32 at 8 x 32^3 20.3 against 55.
        WslabArgs slab{};
        if (static_cast<uint64_t>(s.x) * s.y * s.z * s.batch >= kWslabMinVoxels && wgrad_slab_plan<CIN, COUT>(s, ctas, slab)) {
            CUtensorMap xs_map, dys_map;
            if (!make_activation_map(&xs_map, x, s, CIN, s.x + 1u, slab.rows, 1) ||
                !make_activation_map(&dys_map, dy, s, COUT, s.x + 1u, slab.rows + 2u, 1))
                return XS_CUDA_ERROR;
            static DeviceOnce slab_configured;
            if (!slab_configured.run([] {
                    return cudaFuncSetAttribute(conv3_wgrad_slab_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSlabMaxSmem));
                }))
                return XS_CUDA_ERROR;
            slab.partial = partial;
            slab.redo = reinterpret_cast<uint32_t*>(partial + static_cast<size_t>(ctas) * count);
            slab.ticket = slab.redo + ctas;
            slab.error = error;
            const uint32_t planes = s.batch * slab.strips * s.z, slab_ctas = std::min(ctas, planes);
            conv3_wgrad_slab_kernel<CIN, COUT><<<slab_ctas, kConvThreads, 1024u + slab.slots * slab.slot_bytes, st>>>(xs_map, dys_map, slab);
            if (check_launch() != XS_OK) return XS_CUDA_ERROR;
            args.redo = slab.redo;
            args.redo_count = slab_ctas;
            args.ticket = slab.ticket;
            // (in place of wgrad_reduce_kernel, both launches together: 16 -> 16 at
            // 64^3 23.7 -> 22.8 us, 32 -> 32 at 8 x 32^3 27.1 -> 29.1)
            conv3_wgrad_kernel<CIN, COUT><<<dim3(ctas, L::sets), kConvThreads, L::total, st>>>(xm, ym, args);
            return check_launch();
        }
    }
    conv3_wgrad_kernel<CIN, COUT><<<dim3(ctas, L::sets), kConvThreads, L::total, st>>>(xm, ym, args);
    if (check_launch() != XS_OK) return XS_CUDA_ERROR;
    wgrad_reduce_kernel<<<(count + 255) / 256, 256, 0, st>>>(partial, ctas, count, dw, accumulate ? 1 : 0);
    return check_launch();
}

XsStatus conv3_wgrad(cudaStream_t st, const VolumeShape& s, int cin, int cout, const __nv_bfloat16* x, const __nv_bfloat16* dy, float* partial,
                     float* dw, bool accumulate, int* error) {
#define XS_WGRAD_CASE(CI, CO) \
    if (cin == CI && cout == CO) return launch_wgrad<CI, CO>(st, s, x, dy, partial, dw, accumulate, error);
    XS_WGRAD_CASE(16, 16) XS_WGRAD_CASE(16, 32) XS_WGRAD_CASE(16, 64)
    XS_WGRAD_CASE(32, 16) XS_WGRAD_CASE(32, 32) XS_WGRAD_CASE(32, 64)
    XS_WGRAD_CASE(64, 16) XS_WGRAD_CASE(64, 32) XS_WGRAD_CASE(64, 64)
#undef XS_WGRAD_CASE
    return XS_INVALID_ARGUMENT;
}

}  // namespace xs

using namespace xs;

extern "C" XsStatus xs_conv3d_weight_grad_bf16(cudaStream_t stream, uint32_t batch, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t in_channels,
                                               uint32_t out_channels, const void* input, const void* output_grad, float* partial,
                                               float* weight_grad, uint32_t accumulate, int* error_flag) {
    if (!input || !output_grad || !partial || !weight_grad) return XS_INVALID_ARGUMENT;
    const VolumeShape s{nx, ny, nz, batch};
    return conv3_wgrad(stream, s, static_cast<int>(in_channels), static_cast<int>(out_channels), static_cast<const __nv_bfloat16*>(input),
                       static_cast<const __nv_bfloat16*>(output_grad), partial, weight_grad, accumulate != 0, error_flag);
}

extern "C" size_t xs_conv3d_weight_grad_scratch_floats(uint32_t batch, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t in_channels,
                                                       uint32_t out_channels) {
    const VolumeShape s{nx, ny, nz, batch};
    return wgrad_partial_floats(s, static_cast<int>(in_channels), static_cast<int>(out_channels));
}

extern "C" XsStatus xs_conv3d_bf16(cudaStream_t stream, uint32_t batch, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t in_channels,
                                   uint32_t out_channels, const void* input, const void* weights, const float* bias, void* output,
                                   uint32_t relu, int* error_flag) {
    if (!input || !weights || !output) return XS_INVALID_ARGUMENT;
    const VolumeShape s{nx, ny, nz, batch};
    return conv3_forward(stream, s, static_cast<int>(in_channels), static_cast<int>(out_channels), static_cast<const __nv_bfloat16*>(input),
                         static_cast<const __nv_bfloat16*>(weights), bias, static_cast<__nv_bfloat16*>(output), relu != 0, error_flag);
}
