// f32 Linear over few tokens, or few tiles, on the tensor cores with f32-level accuracy:
//   out[M, N] = X[M, K] . W[N, K]^T (+ bias), everything f32.
//
// ratchet runs f32 models (Phi-2 and Whisper checkpoints as shipped, ops/matmul/gemm.rs) and its CPU
// device, the parity target, accumulates f32 products (cpu/gemm.rs); the bar for f32 ops is 1e-4.
//
// Precision.  Every operand is the sum of three bf16 numbers: its upper half, the rounding of what is left, and the rounding of what is
// left then (24 bits).  Of the nine partial products the six that are not below 2^-23 of the result are taken.  The tensor core adds into its
// accumulator with truncation, always toward zero; so the products of the leading parts and the five small ones have accumulators of their
// own, all start anew every 256 of K (sixteen steps), and the pieces are added up in registers by ordinary rounded additions.  Against 64
// bits, N(0, 1) x N(0, 0.02), relative (this kernel / split-TF32 of gemm_tc_f32.cu or, below 32 tokens, FFMA): 16 x 3072 x 3072 2.3e-7 / 9.9e-7,
// 64 x 2560 x 10240 2.4e-7 / 1.4e-6, 1500 x 384 x 384 2.1e-7 / 5.0e-7.
//
// Structure.  The weights are the 128-row operand and live in tensor memory, the tokens (16, 32 or 64 of a tile) the other one:
//   warp 0       TMA: 128 x 64 f32 of W and T x 64 of X per unit into a ring, 128-byte swizzle;
//   warps 10-25  split both: W's parts go to tensor memory, so that the products read only the tokens from shared memory - with both
//                operands there the split-TF32 kernel is bound by its 128 bytes a cycle (0.7 us for 32 of K); X's parts to swizzled tiles;
//   warp 1       three products per 16 of K, not six: the tokens' parts b1, b2, b3 lie behind one another, so that a1 [b1 b2 b3], a2 [b1 b2] and
//                a3 [b1] are products of 3 T, 2 T and T columns, into three accumulators (a product of 64 columns or fewer costs as
//                much as one of 128, about 64 cycles: one by one the six took 1900 cycles per unit, these 900);
//   warps 2-9    add the accumulators up, a row of W (an output feature) and half of the tokens per thread, and store: 32 consecutive features per token.
// The kernel is persistent.  Tiles are walked whole, or - where they would leave SMs idle - the line of all units (tile, 64 of K) is cut into
// equal runs, one per SM; tiles that are cut leave partial sums which sum_runs_kernel adds in order (deterministic).
//
// What bounds it: the splitting warps (5.5 instructions an element, 70 % of the issue slots), at about 1 us per unit and SM; the bytes of W
// alone would take 0.73.  Measured on B200 (us, before -> now): 2 x 3072 x 3072 204 (FFMA) -> 13, 31 x 3072 x 3072 204 -> 15, 64 x 10240 x 2560
// 49 -> 33, 64 x 2560 x 10240 39 -> 33, 300 x 300 x 1024 25 -> 11, 1500 x 384 x 384 13 -> 10, 2 x 65536 x 1024 412 -> 63.
// Every wait is bounded.
#include <algorithm>

#include "tc_common.cuh"

namespace {

using namespace tc;

constexpr int kUnitK = 64;               // K of a unit
constexpr int kChunk = 4;                // units after which the accumulators start anew
constexpr int kRowsW = 128;              // weight rows of a tile
constexpr int kSumWarps = 8, kConvWarps = 16, kConv0 = 2 + kSumWarps;      // first converting warp
constexpr int kThreadsF32 = (kConv0 + kConvWarps) * 32;
constexpr int kBoxW = kRowsW * 128;      // bytes of 32 columns of a W tile
constexpr int ring_stages(int t) { return t == 64 ? 3 : 4; }
constexpr int stage_bytes(int t) { return 2 * (kBoxW + t * 128); }
constexpr int plane_bytes(int t) { return t * 128; }      // one part of a token tile
constexpr size_t smem_bytes(int t) { return 1024 + (size_t)ring_stages(t) * stage_bytes(t) + (size_t)6 * plane_bytes(t); }

// Cuts the problem: `units` = tiles x nk; runs == 0: CTAs take whole tiles in turn
struct Cut {
    int nk, tiles, tiles_m, tiles_n, runs;
    __device__ __forceinline__ long long units() const { return (long long)tiles * nk; }
    __device__ __forceinline__ long long run_start(int c) const { return units() * c / runs; }
    __device__ __forceinline__ int run_of(long long u) const {
        const long long a = (u + 1) * runs - 1, b = units();
        return a <= 0xffffffffll ? (int)((uint32_t)a / (uint32_t)b) : (int)(a / b);      // a 64-bit division takes a hundred instructions
    }
};

// the segments of this CTA: (tile, first unit, units)
struct Walk {
    const Cut& cut;
    long long u, end;
    int tile, k0, n;
    __device__ __forceinline__ explicit Walk(const Cut& c) : cut(c) {
        if (c.runs) {
            u = c.run_start(blockIdx.x);
            end = c.run_start(blockIdx.x + 1);
        } else {
            u = (long long)blockIdx.x * c.nk;
            end = c.units();
        }
        n = 0;
    }
    __device__ __forceinline__ bool next() {
        if (u >= end) return false;
        tile = (int)(u / cut.nk);
        k0 = (int)(u - (long long)tile * cut.nk);
        n = cut.nk - k0;
        if (cut.runs) {
            if (end - u < n) n = (int)(end - u);
            u += n;
        } else {
            u += (long long)gridDim.x * cut.nk;
        }
        return true;
    }
};

// Two values into their three parts, packed (the first in the lower half).  An infinity is its own leading part and leaves NaN for the others, as
// NaN does: main_and_small has the rest.  (cvt keeps a NaN whose payload lies in the bits that are cut off; taking the upper halves with
// __byte_perm would make an infinity of it for 1 %: 32.4 against 32.0 us for 64 x 2560 x 10240.)
__device__ __forceinline__ void split3(float x, float y, uint32_t (&p)[3]) {
    asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(p[0]) : "f"(y), "f"(x));
    x -= __uint_as_float(p[0] << 16);
    y -= __uint_as_float(p[0] & 0xffff0000u);
    const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
    p[1] = *reinterpret_cast<const uint32_t*>(&b);
    x -= __uint_as_float(p[1] << 16);
    y -= __uint_as_float(p[1] & 0xffff0000u);
    const __nv_bfloat162 c = __floats2bfloat162_rn(x, y);
    p[2] = *reinterpret_cast<const uint32_t*>(&c);
}

// GROUP: the problems share their activations; the others' weights, biases and outputs
template <bool GROUP> struct PartsGroup {};
template <> struct PartsGroup<true> {
    CUtensorMap w[kGroupLinears - 1];
    float* out[kGroupLinears - 1];
    const float* bias[kGroupLinears - 1];
};

// T: tokens of a tile.  RESID: a residual is added behind the bias (a form of its own: 64 x 2560 x 10240 without one stays as it is)
template <int T, bool GROUP = false, bool RESID = false>
__global__ void __launch_bounds__(kThreadsF32, 1)
gemm_parts_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const float* __restrict__ bias,
                const float* __restrict__ bias_rows, const float* __restrict__ resid, float* __restrict__ out, float* __restrict__ partial, int M, int N, const Cut cut, int* status, const __grid_constant__ PartsGroup<GROUP> group) {
    constexpr int R = ring_stages(T), STAGE = stage_bytes(T), PLANE = plane_bytes(T);
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    unsigned char* planes = ring + R * STAGE;            // [2][part]
    __shared__ __align__(8) uint64_t raw_full[R], raw_empty[R], conv_full[2], conv_empty[2], acc_full[2], acc_empty[2], drained;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int i = 0; i < R; ++i) {
            mbar_init(&raw_full[i], 1);
            mbar_init(&raw_empty[i], kConvWarps);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&conv_full[i], kConvWarps);
            mbar_init(&conv_empty[i], 1);
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], kSumWarps);
        }
        mbar_init(&drained, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "n"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    rcu_kernel_entry_wait_only();        // nothing before this touches global memory
    // columns: accumulators a1 b1 | a1 b2 + a2 b1 + a3 b1 | a1 b3 + a2 b2 of T each (twice where they fit), then at 256 two buffers of W's parts
    // (32 columns each)
    constexpr int ACCS = T == 64 ? 1 : 2;
    const uint32_t tmem = tmem_slot;
    Walk walk(cut);

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            while (ok && walk.next()) {
                const int mt = walk.tile % cut.tiles_m, rest = walk.tile / cut.tiles_m, nt = rest % cut.tiles_n;
                int b = rest / cut.tiles_n;
                const CUtensorMap* wm = &wmap;
                if constexpr (GROUP) {
                    if (b > 0) wm = &group.w[b - 1];
                    b = 0;
                }
                for (int k = walk.k0; k < walk.k0 + walk.n; ++k, ++it) {
                    const int s = it % R;
                    if (it >= R && !mbar_wait(&raw_empty[s], (it / R - 1) & 1, &abort_flag, status)) { ok = false; break; }
                    unsigned char* st = ring + s * STAGE;
                    mbar_expect_tx(&raw_full[s], STAGE);
                    for (int h = 0; h < 2; ++h) {
                        tma_load_3d(st + h * kBoxW, wm, k * kUnitK + h * 32, nt * kRowsW, b, &raw_full[s]);
                        tma_load_3d(st + 2 * kBoxW + h * T * 128, &xmap, k * kUnitK + h * 32, mt * T, b, &raw_full[s]);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // the whole warp keeps step, one elected lane issues
        const uint32_t idesc[3] = {umma_idesc_f16(kRowsW, 3 * T, true), umma_idesc_f16(kRowsW, 2 * T, true), umma_idesc_f16(kRowsW, T, true)};
        const uint64_t xd = umma_desc_sw128(planes);
        const bool leader = elect_one();
        auto wait = [&](uint64_t* bar, int phase) { return (bool)__all_sync(0xffffffffu, mbar_wait_spin(bar, phase & 1, &abort_flag, status)); };
        int it = 0, chunk = 0;
        bool ok = true;
        while (ok && walk.next()) {
            for (int i = 0; i < walk.n; ++i, ++it) {
                const int b = it & 1, c = chunk % ACCS;
                const bool first = i % kChunk == 0, last = i % kChunk == kChunk - 1 || i + 1 == walk.n;
                ok = wait(&conv_full[b], it >> 1);
                if (ok && first && chunk >= ACCS) ok = wait(&acc_empty[c], chunk / ACCS - 1);
                if (!ok) break;
                tc_fence_after();
                if (leader) {
                    const uint32_t acc = tmem + (uint32_t)(c * 3 * T), ta = tmem + 256 + (uint32_t)(b * 96);
                    const uint64_t bd = xd + (uint64_t)(b * 3 * (PLANE >> 4));
#pragma unroll
                    for (int k = 0; k < kUnitK / 16; ++k)
#pragma unroll
                        for (int p = 0; p < 3; ++p) umma_f16_ta(acc + (p ? T : 0), ta + 32 * p + 8 * k, bd + 2 * k, idesc[p], !first || k > 0 || p > 0 ? 1u : 0u);
                    umma_commit(&conv_empty[b]);
                    if (last) umma_commit(&acc_full[c]);
                }
                __syncwarp();
                if (last) ++chunk;
            }
        }
        if (!ok && leader) {            // given up: let the products in flight end before tensor memory is freed
            umma_commit(&drained);
            for (int i = 0; i < (1 << 20) && !gemvq8::mbar_test_wait(&drained, 0); ++i) {}
        }
        __syncwarp();
    } else if (warp < kConv0) {
        constexpr int C = T / 2;                                              // tokens of this warp
        const int quarter = warp & 3, row = quarter * 32 + lane, j0 = (warp - 2) / 4 * C;
        const uint32_t t = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)j0;
        int chunk = 0;
        bool ok = true;
        while (ok && walk.next()) {
            float acc[C];
#pragma unroll
            for (int j = 0; j < C; ++j) acc[j] = 0.f;
            for (int i = 0; i < walk.n && ok; i += kChunk, ++chunk) {
                const int c = chunk % ACCS;
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[c], (chunk / ACCS) & 1, &abort_flag, status));
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int j = 0; j < C; j += 8) {
                    float x[8], y[8], z[8];
                    const uint32_t at = t + (uint32_t)(c * 3 * T + j);
                    tmem_ld_32x8(at, x);
                    tmem_ld_32x8(at + T, y);
                    tmem_ld_32x8(at + 2 * T, z);
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[j + e] += main_and_small(x[e], y[e] + z[e]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[c]);
            }
            if (!ok) break;
            const int mt = walk.tile % cut.tiles_m, rest = walk.tile / cut.tiles_m, nt = rest % cut.tiles_n;
            const size_t b = rest / cut.tiles_n;
            const int m0 = mt * T + j0, n = nt * kRowsW + row;
            if (walk.n == cut.nk) {
                if (n < N) {
                    const float* bs = bias;
                    float* ys = out + b * M * N;
                    if constexpr (GROUP) {
                        bs = b > 0 ? group.bias[b - 1] : bias;
                        ys = b > 0 ? group.out[b - 1] : out;
                    }
                    const float bn = bs ? bs[n] : 0.f;
                    float* o = ys + (size_t)m0 * N + n;
                    if constexpr (RESID) {
                        // in batches of sixteen: all 32 of a tile of 64 tokens at once, beside its sums, spilled 188 bytes of a thread beyond its 72 registers
                        // (four of 65 x 9216 x 256 and three products of their results: 77 us, 56 now); eight at a time wait for memory twice as often (69)
                        constexpr int B = 16;
                        static_assert(C % B == 0, "");
                        const float* rs = resid + (size_t)m0 * N + n;
#pragma unroll
                        for (int j0 = 0; j0 < C; j0 += B) {
                            float r[B];
#pragma unroll
                            for (int j = 0; j < B; ++j) r[j] = m0 + j0 + j < M ? rs[(size_t)(j0 + j) * N] : 0.f;
#pragma unroll
                            for (int j = 0; j < B; ++j)
                                if (m0 + j0 + j < M) o[(size_t)(j0 + j) * N] = (acc[j0 + j] + bn) + r[j];
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < C; ++j)
                            if (m0 + j < M) o[(size_t)j * N] = acc[j] + (bias_rows ? bias_rows[m0 + j] : bn);
                    }
                }
            } else {
                float* o = partial + (size_t)(blockIdx.x + walk.tile) * (T * kRowsW) + j0 * kRowsW + row;      // every segment has a place of its own
#pragma unroll
                for (int j = 0; j < C; ++j) o[j * kRowsW] = acc[j];
            }
        }
    } else {
        // waits that suspend (mbar_wait), not mbar_wait_spin: two dozen polling warps took half of the issue slots that the splitting needs
        // a warp splits 16 of the unit's K for 32 rows of W
        const int quarter = warp & 3, group = (warp - kConv0) >> 2, row = quarter * 32 + lane, tid = threadIdx.x - kConv0 * 32;
        const uint32_t ta = tmem + 256 + ((uint32_t)(quarter * 32) << 16) + 8 * group;
        int it = 0;
        bool ok = true;
        while (ok && walk.next()) {
            for (int i = 0; i < walk.n; ++i, ++it) {
                const int s = it % R, b = it & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(&raw_full[s], (it / R) & 1, &abort_flag, status));
                if (ok && it >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&conv_empty[b], ((it >> 1) - 1) & 1, &abort_flag, status));
                if (!ok) break;
                tc_fence_after();
                const unsigned char* st = ring + s * STAGE;
                const unsigned char* line = st + (group >> 1) * kBoxW + row * 128;
                uint32_t p[3][8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = *reinterpret_cast<const float4*>(line + ((((group & 1) * 4 + c) ^ (row & 7)) << 4));
                    uint32_t lo[3], hi[3];
                    split3(v.x, v.y, lo);
                    split3(v.z, v.w, hi);
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        p[q][2 * c] = lo[q];
                        p[q][2 * c + 1] = hi[q];
                    }
                }
#pragma unroll
                for (int q = 0; q < 3; ++q) tmem_st_32x8_start(ta + (uint32_t)(b * 96 + 32 * q), p[q]);
                // tokens: eight values a task, sixteen bytes of each part
                const unsigned char* xs = st + 2 * kBoxW;
                unsigned char* dst = planes + b * 3 * PLANE;
                if (T == 64 || tid < T * 8) {
                    const int r = tid >> 3, c = tid & 7;
                    const unsigned char* src = xs + (c >> 2) * T * 128 + r * 128;
                    const float4 v0 = *reinterpret_cast<const float4*>(src + (((2 * (c & 3)) ^ (r & 7)) << 4)),
                                 v1 = *reinterpret_cast<const float4*>(src + (((2 * (c & 3) + 1) ^ (r & 7)) << 4));
                    uint32_t a0[3], a1[3], a2[3], a3[3];
                    split3(v0.x, v0.y, a0);
                    split3(v0.z, v0.w, a1);
                    split3(v1.x, v1.y, a2);
                    split3(v1.z, v1.w, a3);
#pragma unroll
                    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(dst + q * PLANE + r * 128 + ((c ^ (r & 7)) << 4)) = make_uint4(a0[q], a1[q], a2[q], a3[q]);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&conv_full[b]);
                    mbar_arrive(&raw_empty[s]);          // every value has been stored, so its load is over
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
    }
}

// a tile that was cut: its runs' sums in order + bias per column / per row.  CTA = (tile, eighth of its tokens); thread = feature and token parity
template <int T, bool RESID>
__global__ void __launch_bounds__(256)
sum_runs_kernel(const float* __restrict__ partial, const float* __restrict__ bias, const float* __restrict__ bias_rows, const float* __restrict__ resid, float* __restrict__ out, int M, int N, const Cut cut) {
    rcu_kernel_entry();
    const int tile = blockIdx.x, first = cut.run_of((long long)tile * cut.nk), last = cut.run_of((long long)(tile + 1) * cut.nk - 1);
    if (first == last) return;
    const int mt = tile % cut.tiles_m, rest = tile / cut.tiles_m, nt = rest % cut.tiles_n;
    const size_t b = rest / cut.tiles_n;
    const int row = threadIdx.x & 127, n = nt * kRowsW + row;
    if (n >= N) return;
    const float bn = bias ? bias[n] : 0.f;
    constexpr int J = T / 16;
    const int j0 = blockIdx.y * (T / 8) + (threadIdx.x >> 7);
    float v[J] = {}, r[J] = {};
    if constexpr (RESID) {
#pragma unroll
        for (int i = 0; i < J; ++i)
            if (mt * T + j0 + 2 * i < M) r[i] = resid[(size_t)(mt * T + j0 + 2 * i) * N + n];
    }
    for (int c = first; c <= last; c += 4) {             // four runs requested before the first is added
        float p[4][J];
#pragma unroll
        for (int d = 0; d < 4; ++d)
#pragma unroll
            for (int i = 0; i < J; ++i) p[d][i] = c + d <= last ? partial[(size_t)(c + d + tile) * (T * kRowsW) + (j0 + 2 * i) * kRowsW + row] : 0.f;
#pragma unroll
        for (int d = 0; d < 4; ++d)
#pragma unroll
            for (int i = 0; i < J; ++i) v[i] += p[d][i];
    }
#pragma unroll
    for (int i = 0; i < J; ++i) {
        const int m = mt * T + j0 + 2 * i;
        if (m >= M) continue;
        const float y = v[i] + (bias_rows ? bias_rows[m] : bn);
        out[b * M * N + (size_t)m * N + n] = RESID ? y + r[i] : y;
    }
}

// [batches, rows, K] f32 row-major, box = 1 x box_rows x 32 elements, 128-byte swizzle
bool make_map_f32_sw128(CUtensorMap* map, const void* base, uint64_t batches, uint64_t rows, uint64_t K, uint32_t box_rows) {
    gemvq8::EncodeTiledFn fn = gemvq8::encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {K, rows, batches};
    cuuint64_t strides[2] = {K * 4, rows * K * 4};
    cuuint32_t box[3] = {32, box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Whole tiles (0), or the line of units cut into a run per SM: in units of the longest CTA, the sums of cut tiles (a launch, their partial
// sums out and in again) counted as kSumUnits
int cut_runs(uint64_t sms, uint64_t tiles, uint64_t nk) {
    constexpr uint64_t kSumUnits = 7;
    const uint64_t units = tiles * nk, whole = (tiles + sms - 1) / sms * nk;
    // no more than sixteen runs of a tile: one thread adds an output's up (64 x 64 x 8192, one tile: 28 us with 128 runs)
    const uint64_t runs = std::min({sms, units, 16 * tiles}), even = (units + runs - 1) / runs + kSumUnits;
    return tiles % sms != 0 && even < whole ? (int)runs : 0;
}

template <int T, bool RESID>
rcu_status launch_f32(rcu_device* dev, const void* w, const void* x, const void* bias, const void* bias_rows, void* y, uint64_t M, uint64_t N, uint64_t K, uint64_t batches, const void* resid = nullptr) {
    CUtensorMap xmap, wmap;
    if (!make_map_f32_sw128(&xmap, x, batches, M, K, T) || !make_map_f32_sw128(&wmap, w, batches, N, K, kRowsW))
        return rcu_fail(dev, RCU_ERR_CUDA, "gemm_parts: cuTensorMapEncodeTiled failed (M=%llu N=%llu K=%llu x%llu)", (unsigned long long)M,
                        (unsigned long long)N, (unsigned long long)K, (unsigned long long)batches);
    Cut cut;
    cut.nk = (int)((K + kUnitK - 1) / kUnitK);
    cut.tiles_m = (int)((M + T - 1) / T);
    cut.tiles_n = (int)((N + kRowsW - 1) / kRowsW);
    const uint64_t tiles = batches * cut.tiles_m * (uint64_t)cut.tiles_n;
    if (tiles > 0x3fffffffull) return RCU_ERR_UNSUPPORTED;
    cut.tiles = (int)tiles;
    const uint64_t sms = dev->sm_count;
    cut.runs = cut_runs(sms, tiles, cut.nk);
    void* partial = nullptr;
    if (cut.runs) {
        if (rcu_alloc(dev, (cut.runs + tiles) * (uint64_t)(T * kRowsW) * 4, &partial) != RCU_OK) cut.runs = 0;      // no room: whole tiles need none
    }
    const unsigned grid = cut.runs ? (unsigned)cut.runs : (unsigned)std::min(tiles, sms);
    auto kern = gemm_parts_kernel<T, false, RESID>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(T));
    if (e == cudaSuccess)
        e = rcu_launch(dev, kern, grid, kThreadsF32, smem_bytes(T), xmap, wmap, (const float*)bias, (const float*)bias_rows, (const float*)resid, (float*)y, (float*)partial, (int)M,
                       (int)N, cut, dev->d_status, PartsGroup<false>{});
    dev->launches++;
    if (e == cudaSuccess && cut.runs) {
        e = rcu_launch(dev, sum_runs_kernel<T, RESID>, dim3((unsigned)tiles, 8), 256, 0, (const float*)partial, (const float*)bias, (const float*)bias_rows, (const float*)resid, (float*)y, (int)M, (int)N, cut);
        dev->launches++;
    }
    if (partial) rcu_free(dev, partial);          // the pool reuses blocks in stream order
    return e == cudaSuccess ? RCU_OK : rcu_fail(dev, RCU_ERR_CUDA, "gemm_parts: %s", cudaGetErrorString(e));
}

}  // namespace

// Products over the same rows as tiles of one launch, whole ones: short K (longer ones are cut into runs by themselves: their sums' order would change) and a
// product's tiles no more than the SMs (beyond that the split-TF32 kernel has them).  Whisper-tiny's three of 1500 x 384 x 384 take one of them 10 us, the encoder with its
// four layers 605 us before and 563 with them together.  Us for four such groups and the products of their results, apart / together: 2 x 200 x 384 x 384 87.5 / 57.8,
// 3 x 750 x 512 x 512 161 / 79, 3 x 2000 x 512 x 384 (128 tiles) 174 / 134.  Beyond the limit on K whole tiles would pay further, up to where
// cutting does: 3 x 300 x 1024 x 1024 190 / 110, 2 x 400 x 512 x 2048 135 / 162.
bool rcu_gemm_tc_f32_eligible(int lhs_dt, int act_dt, uint64_t M, uint64_t N, uint64_t K, uint64_t batches);
rcu_status rcu_gemm_parts_f32_group(rcu_device* dev, const LinearGroup& g) {
    constexpr int T = 64;
    if (g.n < 2 || g.n > kGroupLinears || g.M <= T || g.K > 8 * kUnitK || g.K < 64 || g.K % 4 || g.N % 4 || g.M > 0x7fffffffull || g.N > 0x7fffffffull || !rcu_gemm_tc_f32_eligible(RCU_F32, RCU_F32, g.M, g.N, g.K, 1))
        return RCU_ERR_UNSUPPORTED;
    const uint64_t tiles_m = (g.M + T - 1) / T, tiles_n = (g.N + kRowsW - 1) / kRowsW, tiles = tiles_m * tiles_n;
    if (tiles > (uint64_t)dev->sm_count) return RCU_ERR_UNSUPPORTED;
    uintptr_t at = (uintptr_t)g.x;
    for (int i = 0; i < g.n; ++i) at |= (uintptr_t)g.w[i] | (uintptr_t)g.out[i];
    if (at & 15) return RCU_ERR_UNSUPPORTED;
    DevGuard guard(dev->ordinal);
    CUtensorMap xmap, wmap;
    PartsGroup<true> group{};
    bool maps = make_map_f32_sw128(&xmap, g.x, 1, g.M, g.K, T) && make_map_f32_sw128(&wmap, g.w[0], 1, g.N, g.K, kRowsW);
    for (int i = 1; i < g.n; ++i) {
        maps = maps && make_map_f32_sw128(&group.w[i - 1], g.w[i], 1, g.N, g.K, kRowsW);
        group.out[i - 1] = (float*)g.out[i];
        group.bias[i - 1] = (const float*)g.bias[i];
    }
    if (!maps) return rcu_fail(dev, RCU_ERR_CUDA, "gemm_parts: cuTensorMapEncodeTiled failed (group, M=%llu N=%llu K=%llu)", (unsigned long long)g.M, (unsigned long long)g.N, (unsigned long long)g.K);
    Cut cut;
    cut.nk = (int)((g.K + kUnitK - 1) / kUnitK);
    cut.tiles_m = (int)tiles_m;
    cut.tiles_n = (int)tiles_n;
    cut.tiles = (int)(tiles * g.n);
    cut.runs = 0;
    const unsigned grid = (unsigned)std::min<uint64_t>(cut.tiles, dev->sm_count);
    auto kern = gemm_parts_kernel<T, true>;
    RCU_CUDA(dev, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(T)));
    RCU_CUDA(dev, rcu_launch(dev, kern, grid, kThreadsF32, smem_bytes(T), xmap, wmap, (const float*)g.bias[0], (const float*)nullptr, (const float*)nullptr, (float*)g.out[0], (float*)nullptr, (int)g.M, (int)g.N,
                             cut, dev->d_status, group));
    RCU_LAUNCH_CHECK(dev);
    return RCU_OK;
}

namespace {
// Up to 64 tokens, and wherever the tiles leave room on the SMs.  With more tiles than that the 128 x 128 tiles of the split-TF32 kernel
// need fewer bytes of shared memory per product (us here / there: 1500 x 1536 x 384, 288 tiles, 20.2 / 16.3; 512 x 3072 x 3072, 192, 74 / 66;
// 1500 x 384 x 1536, 72, 21.3 / 23.3; 128 x 3072 x 3072, 48, 25.1 / 26.2; 64 x 10240 x 2560 33 / 49).  Rows that do not start on four columns
// come here at any size: the FMA pipe, which they would go to otherwise, is as exact as this and the split-TF32 kernel is not.
bool takes(rcu_device* dev, uint64_t M, uint64_t N, uint64_t batches) {
    const uint64_t tiles = batches * ((M + 63) / 64) * ((N + kRowsW - 1) / kRowsW);
    return M <= 64 || N % 4 != 0 || tiles <= (uint64_t)dev->sm_count;
}
rcu_status dispatch(rcu_device* dev, const void* w, const void* x, const void* bias, void* y, uint64_t M, uint64_t N, uint64_t K, uint64_t batches, const void* bias_rows,
                    const void* resid) {
    // Tiles of 32 tokens where they leave room on the SMs too and K is short: a CTA's chain of units is what counts then, and theirs are shorter
    // (33 x 64 x 256: 9.8 us with tiles of 64)
    const bool narrow = K <= 8 * kUnitK && batches * ((M + 31) / 32) * ((N + kRowsW - 1) / kRowsW) <= (uint64_t)dev->sm_count;
    if (resid) return narrow ? launch_f32<32, true>(dev, w, x, bias, bias_rows, y, M, N, K, batches, resid) : launch_f32<64, true>(dev, w, x, bias, bias_rows, y, M, N, K, batches, resid);
    if (M <= 16) return launch_f32<16, false>(dev, w, x, bias, bias_rows, y, M, N, K, batches);
    if (M <= 32 || narrow) return launch_f32<32, false>(dev, w, x, bias, bias_rows, y, M, N, K, batches);
    return launch_f32<64, false>(dev, w, x, bias, bias_rows, y, M, N, K, batches);
}
}  // namespace

// RCU_ERR_UNSUPPORTED: gemm_tc_f32.cu's kernel is the faster one
rcu_status rcu_gemm_parts_f32_dispatch(rcu_device* dev, const void* w, const void* x, const void* bias, void* y, uint64_t M, uint64_t N, uint64_t K, uint64_t batches,
                                       const void* bias_rows) {
    return takes(dev, M, N, batches) ? dispatch(dev, w, x, bias, y, M, N, K, batches, bias_rows, nullptr) : RCU_ERR_UNSUPPORTED;
}

// The residual too, where that is no slower than an addition behind the product: tiles that are cut into runs (whose sums are a pass over the output anyway) and short
// K.  Whole tiles of longer K wait for it with their SM to themselves (us for four of them and three products, apart / in: 65 x 768 x 768 52.1 / 45.1, 1500 x 384 x 384
// 54.2 / 49.4, 1500 x 512 x 512 72.2 / 70.5, 65 x 9216 x 256 55.8 / 55.8, 750 x 768 x 768 86.2 / 86.2, 750 x 1024 x 1024 105.0 / 107.6, 129 x 4096 x 1024 104.2 / 108.5).
bool rcu_gemm_parts_f32_takes(rcu_device* dev, uint64_t M, uint64_t N, uint64_t K) {
    if (!rcu_gemm_tc_f32_eligible(RCU_F32, RCU_F32, M, N, K, 1) || !takes(dev, M, N, 1)) return false;
    return K <= 8 * kUnitK || cut_runs(dev->sm_count, (M + 63) / 64 * ((N + kRowsW - 1) / kRowsW), (K + kUnitK - 1) / kUnitK) > 0;
}
rcu_status rcu_gemm_parts_f32_resid(rcu_device* dev, const void* w, const void* x, const void* bias, const void* resid, void* y, uint64_t M, uint64_t N, uint64_t K) {
    if (!rcu_gemm_parts_f32_takes(dev, M, N, K)) return RCU_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(bias)) & 15) return RCU_ERR_UNSUPPORTED;
    DevGuard g(dev->ordinal);
    return dispatch(dev, w, x, bias, y, M, N, K, 1, nullptr, resid);
}
