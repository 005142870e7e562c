// Attention of an f32 prompt on the 5th-generation tensor cores with f32-level accuracy: what a graph of the form
//   softmax((dk q) (dk k)^T) v        (whisper/mha.rs:92-127)
// asks for, without its score matrices in memory.  The resolver (graph_fusion.cuh) sends such subgraphs here.
//
// Precision.  Every f32 operand is the sum of three bf16 numbers (rounding, rounding of the remainder, and again: 24 bits), and a
// product takes the six of the nine partial products that are not below 2^-24 of the result.  Tensor cores add into their accumulator
// with truncation, so the products of the leading parts and the five small ones go to accumulators of their own, each of which starts anew
// at every tile of 64 keys (four steps); the sums over the tiles are ordinary rounded f32 arithmetic in registers, as are scores, maxima
// and weights (expf).  Measured against 64 bits (6 heads of 64, 1500 positions): relative error 3.8e-7, where the chain of split-TF32
// products and the f32 softmax has 1.6e-6.
//
// Structure.  split_heads_kernel brings q, k and v (strided views of the projections, with their factors) into planes
// [part][head][position][64] that TMA can read.  attention_f32_kernel: CTA = 256 queries of one head and a run of key tiles; two tiles of 128
// queries take turns as in attention_tc.cu, S and the weights' three parts share tensor memory, O of a tile is added up by the thread that
// holds the query.  Runs of keys are split over CTAs until the SMs are covered (36 CTAs otherwise for 6 heads of 1500 positions) and
// merged by merge_kernel.
//
// What bounds it: the softmax warps (some thirty instructions a score: sum of two accumulators, maximum, expf, three roundings), about as
// long as the 48 products of a tile; splitting and merging move 25 MB through L2.  Measured on B200, the encoder of Whisper-tiny over 3000
// frames (four layers of 6 heads, 1500 positions): 1041 -> 695 us, of which the eleven kernels per layer that this replaces took 575.
// Every wait is bounded; one that gives up raises RCU_DEVFLAG_TIMEOUT and ends all others of the CTA.
#include <cuda.h>

#include "attention.cuh"
#include "tc_common.cuh"

namespace {

using namespace tc;

constexpr int kTileQ = 128, kTileK = 64, kCols = 64, kThreadsA = 320;
constexpr int kBlockQ = kTileQ * 128, kBlockK = kTileK * 128;       // bytes of one part of a query / key tile

struct SplitArgs {
    const float* x[3];
    size_t head[3], row[3];
    int rows[3], cols[3];
    const float* scale[3];       // one factor, nullable
    __nv_bfloat16* planes[3];    // [3][H][rows][64]
    int H;
};

// thread = eight features of one (position, head) of one operand
__global__ void __launch_bounds__(256) split_heads_kernel(const __grid_constant__ SplitArgs a) {
    rcu_kernel_entry();
    const int w = blockIdx.y, rows = a.rows[w], cols = a.cols[w];
    const size_t n = (size_t)rows * a.H * 8;
    const float f = a.scale[w] ? *a.scale[w] : 1.f;
    const size_t plane = (size_t)a.H * rows * kCols;
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
        const int c = (int)(i & 7) * 8;
        const size_t th = i >> 3, t = th / a.H, h = th - t * a.H;
        const float* src = a.x[w] + h * a.head[w] + t * a.row[w] + c;
        float v[8] = {};
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (c + 4 * q < cols) *reinterpret_cast<float4*>(v + 4 * q) = *reinterpret_cast<const float4*>(src + 4 * q);      // cols is a multiple of 4
        __align__(16) __nv_bfloat16 p[3][8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            float x = a.scale[w] ? __fmul_rn(v[e], f) : v[e];
            __nv_bfloat16 top = __float2bfloat16_rn(x);
            if (isinf(__bfloat162float(top))) top = __ushort_as_bfloat16((unsigned short)(__float_as_uint(x) >> 16));      // finite x stays finite
            p[0][e] = top;
            x -= __bfloat162float(top);
            p[1][e] = __float2bfloat16_rn(x);
            p[2][e] = __float2bfloat16_rn(x - __bfloat162float(p[1][e]));
        }
        __nv_bfloat16* dst = a.planes[w] + (h * rows + t) * kCols + c;
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint4*>(dst + k * plane) = *reinterpret_cast<const uint4*>(p[k]);
    }
}

struct Args {
    float* out;          // [T][H][E], or unnormalised partial sums [run][T][H][E]
    float2* ml;          // [run][T][H]: maximum and sum of the weights; null: one run
    int H, T, L, E;
    int tiles_per_run;
    int* status;
};

// CARE: infinite operands give what f32 arithmetic gives (main_and_small), not NaN
template <bool CARE>
__global__ void __launch_bounds__(kThreadsA, 1)
attention_f32_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, const Args a) {
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* qs = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);      // [tile][part]
    unsigned char* ks = qs + 6 * kBlockQ;               // [stage][part]
    unsigned char* vs = ks + 6 * kBlockK;
    __shared__ __align__(8) uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], pv_done[2], drained;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.x, i0 = blockIdx.y * 2 * kTileQ;
    const int nq = min(2 * kTileQ, a.T - i0);
    const int first = blockIdx.z * a.tiles_per_run, tiles = min(a.tiles_per_run, (a.L + kTileK - 1) / kTileK - first);      // at least one
    const bool second = nq > kTileQ;

    if (threadIdx.x == 0) {
        mbar_init(&q_full, 1);
        mbar_init(&drained, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 4);
            mbar_init(&pv_done[i], 1);
        }
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
    // per query tile 256 columns: S of the leading parts 64, S of the small products 64 (the weights' parts, 32 columns each, take their
    // place), O of the leading parts 64, O of the small products 64
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(&q_full, 6 * kBlockQ);       // rows beyond T arrive as zeros
            for (int w = 0; w < 2; ++w)
                for (int p = 0; p < 3; ++p) tma_load_3d(qs + (w * 3 + p) * kBlockQ, &qmap, 0, i0 + w * kTileQ, p * a.H + h, &q_full);
            for (int n = 0; n < tiles; ++n) {
                const int s = n & 1, ph = ((n >> 1) - 1) & 1, j0 = (first + n) * kTileK;
                if (n >= 2 && !mbar_wait(&k_empty[s], ph, &abort_flag, a.status)) break;
                mbar_expect_tx(&k_full[s], 3 * kBlockK);
                for (int p = 0; p < 3; ++p) tma_load_3d(ks + (s * 3 + p) * kBlockK, &kmap, 0, j0, p * a.H + h, &k_full[s]);
                if (n >= 2 && !mbar_wait(&v_empty[s], ph, &abort_flag, a.status)) break;
                mbar_expect_tx(&v_full[s], 3 * kBlockK);
                for (int p = 0; p < 3; ++p) tma_load_3d(vs + (s * 3 + p) * kBlockK, &vmap, 0, j0, p * a.H + h, &v_full[s]);
            }
        }
    } else if (warp == 1) {
        // the whole warp keeps step, one elected lane issues
        const uint32_t idesc_s = umma_idesc_f16(kTileQ, kTileK, true);
        const uint32_t idesc_o = umma_idesc_f16(kTileQ, kCols, true) | (1u << 16);          // V is stored with its columns contiguous
        const uint64_t qd = umma_desc_sw128(qs), kd = umma_desc_sw128(ks), vd = umma_desc_sw128_mn(vs, kBlockK);
        const bool leader = elect_one();
        auto wait = [&](uint64_t* bar, int phase) { return (bool)__all_sync(0xffffffffu, mbar_wait_spin(bar, phase & 1, &abort_flag, a.status)); };
        // S of key tile n for query tile w
        auto scores = [&](int w, int n) {
            if (leader) {
                const uint32_t t = tmem + (uint32_t)w * 256;
                const uint64_t ad = qd + (uint64_t)(w * 3 * (kBlockQ >> 4)), bd = kd + (uint64_t)((n & 1) * 3 * (kBlockK >> 4));
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int p = 2; p >= 0; --p)
#pragma unroll
                        for (int q = 2 - p; q >= 0; --q) {
                            const bool main = p == 0 && q == 0;
                            umma_f16(t + (main ? 0 : 64), ad + p * (kBlockQ >> 4) + 2 * k, bd + q * (kBlockK >> 4) + 2 * k, idesc_s,
                                     k > 0 || !(main || (p == 2 && q == 0)) ? 1u : 0u);
                        }
                umma_commit(&s_full[w]);
            }
            __syncwarp();
        };
        bool ok = wait(&q_full, 0);
        if (ok) ok = wait(&k_full[0], 0);
        tc_fence_after();
        if (ok) {
            scores(0, 0);
            if (second) scores(1, 0);
            if (leader) umma_commit(&k_empty[0]);
            __syncwarp();
        }
        for (int n = 0; n < tiles && ok; ++n) {
            const int s = n & 1;
            const bool more = n + 1 < tiles;
            ok = wait(&v_full[s], n >> 1);
            if (ok && more) ok = wait(&k_full[s ^ 1], (n + 1) >> 1);
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                if (!ok || (w == 1 && !second)) continue;
                ok = wait(&p_full[w], n);
                if (!ok) continue;
                tc_fence_after();
                if (leader) {
                    const uint32_t t = tmem + (uint32_t)w * 256;
                    const uint64_t bd = vd + (uint64_t)(s * 3 * (kBlockK >> 4));
#pragma unroll
                    for (int k = 0; k < kTileK / 16; ++k)          // 16 keys are two 1024-byte groups of V, eight columns of a part of P
#pragma unroll
                        for (int p = 2; p >= 0; --p)
#pragma unroll
                            for (int q = 2 - p; q >= 0; --q) {
                                const bool main = p == 0 && q == 0;
                                umma_f16_ta(t + (main ? 128 : 192), t + 32 * p + 8 * k, bd + q * (kBlockK >> 4) + 128 * k, idesc_o,
                                            k > 0 || !(main || (p == 2 && q == 0)) ? 1u : 0u);
                            }
                    umma_commit(&pv_done[w]);
                }
                __syncwarp();
                if (more) {                                         // the next scores take the place of these weights
                    ok = wait(&pv_done[w], n);
                    tc_fence_after();
                    if (ok) scores(w, n + 1);
                }
            }
            if (!ok) break;
            if (leader) {
                umma_commit(&v_empty[s]);
                if (more) umma_commit(&k_empty[s ^ 1]);
            }
            __syncwarp();
        }
        if (!ok && leader) {            // given up: let the products in flight end before tensor memory is freed
            umma_commit(&drained);
            for (int i = 0; i < (1 << 20) && !gemvq8::mbar_test_wait(&drained, 0); ++i) {}
        }
        __syncwarp();
    } else if (warp < 6 || second) {
        const int w = warp < 6 ? 0 : 1, quarter = warp & 3;
        const int r = w * kTileQ + quarter * 32 + lane;                        // query of the CTA
        const uint32_t t = tmem + (uint32_t)w * 256 + ((uint32_t)(quarter * 32) << 16);
        float acc[kCols], m = -INFINITY, l = 0.f, corr = 0.f;
#pragma unroll
        for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
        // acc = acc * corr + O of the tile whose weights were written last
        auto add_tile = [&]() {
#pragma unroll
            for (int c = 0; c < kCols; c += 32) {
                float x[32], y[32];
                tmem_ld_32x32(t + 128 + c, x);
                tmem_ld_32x32(t + 192 + c, y);
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[c + j] = fmaf(acc[c + j], corr, CARE ? main_and_small(x[j], y[j]) : x[j] + y[j]);
            }
        };
        bool ok = true;
        for (int n = 0; n < tiles; ++n) {
            if (n > 0) {                                                      // while the tensor cores are at the next scores
                ok = __all_sync(0xffffffffu, mbar_wait_spin(&pv_done[w], (n - 1) & 1, &abort_flag, a.status));
                if (!ok) break;
                tc_fence_after();
                add_tile();
            }
            ok = __all_sync(0xffffffffu, mbar_wait_spin(&s_full[w], n & 1, &abort_flag, a.status));
            if (!ok) break;
            tc_fence_after();
            float s[kTileK];
#pragma unroll
            for (int c = 0; c < kTileK; c += 32) {
                float y[32];
                tmem_ld_32x32(t + c, s + c);
                tmem_ld_32x32(t + 64 + c, y);
#pragma unroll
                for (int j = 0; j < 32; ++j) s[c + j] = CARE ? main_and_small(s[c + j], y[j]) : s[c + j] + y[j];
            }
            const int left = a.L - (first + n) * kTileK;
            if (left < kTileK) {
#pragma unroll
                for (int j = 0; j < kTileK; ++j)
                    if (j >= left) s[j] = -INFINITY;
            }
            float top4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
            for (int j = 4; j < kTileK; ++j) top4[j & 3] = fmaxf(top4[j & 3], s[j]);
            const float next = fmaxf(m, fmaxf(fmaxf(top4[0], top4[1]), fmaxf(top4[2], top4[3])));
            corr = m == next ? 1.f : expf(m - next);                          // 0 while no key has been seen
            m = next;
            const float z = m == -INFINITY ? 0.f : m;
            float l4[4] = {l * corr, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < kTileK; c += 32) {                            // 32 keys are 16 columns of each part
                uint32_t part[3][16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float x = expf(s[c + 2 * j] - z), y = expf(s[c + 2 * j + 1] - z);
                    l4[j & 3] += x + y;
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
                        part[p][j] = *reinterpret_cast<const uint32_t*>(&b);
                        x -= __uint_as_float(part[p][j] << 16);
                        y -= __uint_as_float(part[p][j] & 0xffff0000u);
                    }
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) tmem_st_32x16(t + 32 * p + c / 2, part[p]);
            }
            l = (l4[0] + l4[1]) + (l4[2] + l4[3]);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[w]);
        }
        if (ok) {
            ok = __all_sync(0xffffffffu, mbar_wait(&pv_done[w], (tiles - 1) & 1, &abort_flag, a.status));
            tc_fence_after();
            if (ok) {
                add_tile();
                if (r < nq) {
                    const size_t th = (size_t)(i0 + r) * a.H + h;
                    float* out = a.out + ((size_t)blockIdx.z * a.T * a.H + th) * a.E;
                    float inv = 1.f;
                    if (a.ml) a.ml[(size_t)blockIdx.z * a.T * a.H + th] = make_float2(m, l);
                    else inv = 1.0f / l;
#pragma unroll
                    for (int j = 0; j < kCols; j += 4)
                        if (j < a.E) *reinterpret_cast<float4*>(out + j) = make_float4(acc[j] * inv, acc[j + 1] * inv, acc[j + 2] * inv, acc[j + 3] * inv);
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

// thread = four features of one (position, head): the runs' sums against the largest of their maxima
__global__ void __launch_bounds__(256)
merge_kernel(const float* __restrict__ part, const float2* __restrict__ ml, float* __restrict__ out, size_t th, int E, int runs) {
    rcu_kernel_entry();
    const int e4 = E / 4;
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < th * e4; i += (size_t)gridDim.x * 256) {
        const size_t r = i / e4, c = (i - r * e4) * 4;
        float m = -INFINITY;
        for (int k = 0; k < runs; ++k) m = fmaxf(m, ml[k * th + r].x);
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        float l = 0.f;
        for (int k = 0; k < runs; ++k) {
            const float2 s = ml[k * th + r];
            const float4 p = *reinterpret_cast<const float4*>(part + (k * th + r) * E + c);
            const float w = expf(s.x - m);
            l = fmaf(w, s.y, l);
            o = make_float4(fmaf(w, p.x, o.x), fmaf(w, p.y, o.y), fmaf(w, p.z, o.z), fmaf(w, p.w, o.w));
        }
        const float inv = 1.0f / l;
        *reinterpret_cast<float4*>(out + r * E + c) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
    }
}

// [3 H][rows][64] bf16, a box of `box_rows` rows, 128-byte swizzle; rows beyond the extent read as zero
bool map_planes(CUtensorMap* map, const void* base, uint64_t heads, uint64_t rows, uint32_t box_rows) {
    gemvq8::EncodeTiledFn fn = gemvq8::encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {kCols, rows, 3 * heads};
    cuuint64_t strides[2] = {kCols * 2, rows * kCols * 2};
    cuuint32_t box[3] = {kCols, box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr size_t kSmem = 1024 + 6 * kBlockQ + 12 * kBlockK;

}  // namespace

bool rcu_f32_tensor_cores();      // gemm_tc_f32.cu

bool rcu_attention_f32_takes(const rcu_device* dev, const Attention32Args& a) {
    if (a.T < 2 || a.L < 1 || a.H < 1 || a.H > 65535 || a.T > 65535 * 2 * kTileQ || a.L > (1 << 30)) return false;
    if (a.D < 4 || a.D > kCols || a.D % 4 || a.E < 4 || a.E > kCols || a.E % 4) return false;
    for (const HeadRows* t : {&a.q, &a.k, &a.v})
        if (t->head % 4 || t->row % 4) return false;
    return rcu_f32_tensor_cores() && kSmem + 1024 <= (size_t)dev->smem_optin;
}

rcu_status rcu_attention_f32(rcu_device* dev, const Attention32Args& a) {
    if (!rcu_attention_f32_takes(dev, a)) return RCU_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(a.q.data) | reinterpret_cast<uintptr_t>(a.k.data) | reinterpret_cast<uintptr_t>(a.v.data) | reinterpret_cast<uintptr_t>(a.out)) & 15)
        return RCU_ERR_UNSUPPORTED;
    DevGuard g(dev->ordinal);
    const uint64_t H = a.H, T = a.T, L = a.L, th = T * H;
    // Runs of keys: as many as cover the SMs, of two tiles at least (a run's partial sums are written and read again)
    const int blocks = (int)(H * ((T + 2 * kTileQ - 1) / (2 * kTileQ))), tiles = (int)((L + kTileK - 1) / kTileK);
    int runs = std::min(std::max(1, dev->sm_count / blocks), std::max(1, tiles / 2));
    const int per = (tiles + runs - 1) / runs;
    runs = (tiles + per - 1) / per;
    const uint64_t q_bytes = 3 * th * kCols * 2, kv_bytes = 3 * L * H * kCols * 2, part_bytes = runs > 1 ? runs * th * a.E * 4 : 0;
    void *planes = nullptr, *part = nullptr;
    rcu_status st = rcu_alloc(dev, q_bytes + 2 * kv_bytes, &planes);
    if (st == RCU_OK && runs > 1) st = rcu_alloc(dev, part_bytes + runs * th * 8, &part);
    if (st != RCU_OK) {
        if (planes) rcu_free(dev, planes);
        return st;
    }
    char* p = (char*)planes;
    SplitArgs s{};
    const HeadRows* src[3] = {&a.q, &a.k, &a.v};
    for (int i = 0; i < 3; ++i) {
        s.x[i] = (const float*)src[i]->data;
        s.head[i] = src[i]->head;
        s.row[i] = src[i]->row;
        s.rows[i] = i ? a.L : a.T;
        s.cols[i] = i == 2 ? a.E : a.D;
        s.scale[i] = i < 2 ? a.scale[i] : nullptr;
        s.planes[i] = (__nv_bfloat16*)(p + (i ? q_bytes + (i - 1) * kv_bytes : 0));
    }
    s.H = a.H;
    CUtensorMap qm, km, vm;
    cudaError_t e = cudaSuccess;
    if (!map_planes(&qm, s.planes[0], H, T, kTileQ) || !map_planes(&km, s.planes[1], H, L, kTileK) || !map_planes(&vm, s.planes[2], H, L, kTileK)) {
        st = rcu_fail(dev, RCU_ERR_CUDA, "attention: cuTensorMapEncodeTiled failed (T=%d L=%d H=%d)", a.T, a.L, a.H);
    } else {
        const Args t{runs > 1 ? (float*)part : (float*)a.out, runs > 1 ? (float2*)((char*)part + part_bytes) : nullptr, a.H, a.T, a.L, a.E, per, dev->d_status};
        e = rcu_launch(dev, split_heads_kernel, dim3((unsigned)grid_for(std::max(T, L) * H * 8, 256, dev->sm_count * 8), 3), 256, 0, s);
        // Fewer than 32 positions have their products on the FMA pipe with one kernel per op, and infinities with them; from 32 on those products
        // are split too and give NaN.  The minimum on every value costs 4 % of the kernel (36.4 us for 35.1, 6 heads of 1500 positions).
        const auto kern = a.T < 32 ? attention_f32_kernel<true> : attention_f32_kernel<false>;
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
        if (e == cudaSuccess)
            e = rcu_launch(dev, kern, dim3(a.H, (a.T + 2 * kTileQ - 1) / (2 * kTileQ), runs), kThreadsA, kSmem, qm, km, vm, t);
        if (e == cudaSuccess && runs > 1)
            e = rcu_launch(dev, merge_kernel, (unsigned)grid_for(th * (a.E / 4), 256, dev->sm_count * 8), 256, 0, (const float*)part, t.ml, (float*)a.out, (size_t)th, a.E, runs);
        dev->launches += runs > 1 ? 3 : 2;
    }
    rcu_free(dev, planes);          // the pool reuses blocks in stream order
    if (part) rcu_free(dev, part);
    if (st == RCU_OK && e != cudaSuccess) st = rcu_fail(dev, RCU_ERR_CUDA, "attention: %s", cudaGetErrorString(e));
    return st;
}
