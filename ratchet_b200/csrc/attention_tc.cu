// Attention of an f16 prompt on the 5th-generation tensor cores (tcgen05): what a graph of the form
//   softmax(scale * q k^T [+ mask]) v        (phi3/attn.rs:120-157, whisper/mha.rs:92-127)
// asks for, in one kernel and without its score matrices in memory.  The resolver (graph_fusion.cuh) sends such subgraphs here.
//
// CTA = 256 queries of one head, in two tiles of 128 that take turns, as in window_tc.cu, or one tile of 128 where few CTAs would be left: TMA
// brings the queries once, then 64 keys, their values and the mask's 256 x 64 piece per stage; one warp issues S = Q K^T and O += P V with P read from tensor memory; eight warps hold a
// query per thread.  With a mask the scores are rounded where the graph rounds them (f16 after the scale, f16 after the mask), so that
// a row whose keys are all masked with the type's lowest value averages over them as it does there; without one they stay f32.
// Weights enter the product in f16, which is the type the graph casts them to; their sum is taken in f32 before that.
//
// What bounds it: the softmax warps (64 scores per thread and key tile: scale, two roundings, maximum, exponential, packing), not the
// products.  Measured on B200, 32 heads of 96, 1000 positions with mask: the twelve kernels it replaces took 430 us per layer.
// Every wait is bounded; one that gives up raises RCU_DEVFLAG_TIMEOUT and ends all others of the CTA.
#include <cuda.h>

#include "attention.cuh"
#include "tc_common.cuh"

rcu_status rcu_copy2d_pitched(rcu_device* dev, const void* src, void* dst, size_t rows, size_t row_bytes, size_t spitch, size_t dpitch);

namespace {

using namespace tc;

constexpr int kTileQ = 128, kTileK = 64, kThreadsA = 320;
constexpr int kBlockQ = kTileQ * 128, kBlockK = kTileK * 128;       // bytes of 64 columns of a query / key tile

struct Args {
    __half* out;
    int H, T, L, E;
    int per;                    // queries of a CTA, one tile or two
    const float* scale32;
    const __half *scale_q, *scale_k;
    int* status;
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// NB: 64-column blocks of a query and a key, EB: of a value; MASK: scores rounded to f16 and a mask added
template <int NB, int EB, bool MASK>
__global__ void __launch_bounds__(kThreadsA, 1)
attention_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                 const __grid_constant__ CUtensorMap mmap, const Args a) {
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* qs = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    unsigned char* ks = qs + 2 * NB * kBlockQ;
    unsigned char* vs = ks + 2 * NB * kBlockK;
    unsigned char* ms = vs + 2 * EB * kBlockK;          // MASK: two stages of two 128 x 64 pieces
    __shared__ __align__(8) uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], m_full[2], m_empty[2], s_full[2][2], p_full[2][2], pv_done[2], drained;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.x, i0 = blockIdx.y * a.per;
    const int nq = min(a.per, a.T - i0);               // the CTA's queries
    const int tiles = (a.L + kTileK - 1) / kTileK;
    const bool second = nq > kTileQ;                        // whether the second query tile holds any

    if (threadIdx.x == 0) {
        mbar_init(&q_full, 1);
        mbar_init(&drained, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
            mbar_init(&m_full[i], 1);
            mbar_init(&m_empty[i], second ? 8 : 4);
            for (int b = 0; b < 2; ++b) {
                mbar_init(&s_full[i][b], 1);
                mbar_init(&p_full[i][b], 4);
            }
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
    const uint32_t tmem = tmem_slot;       // per query tile 256 columns: two buffers of 64 (S, then P), 128 for O

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(&q_full, 2 * NB * kBlockQ);
            for (int w = 0; w < 2; ++w)
                for (int b = 0; b < NB; ++b) tma_load_3d(qs + (w * NB + b) * kBlockQ, &qmap, b * 64, h, i0 + w * kTileQ, &q_full);
            // keys (and the mask) run one tile ahead of values
            for (int n = 0; n <= tiles; ++n) {
                if (n < tiles) {
                    const int s = n & 1, j0 = n * kTileK, ph = ((n >> 1) - 1) & 1;
                    if (n >= 2 && !mbar_wait(&k_empty[s], ph, &abort_flag, a.status)) break;
                    mbar_expect_tx(&k_full[s], NB * kBlockK);
                    for (int b = 0; b < NB; ++b) tma_load_3d(ks + (s * NB + b) * kBlockK, &kmap, b * 64, h, j0, &k_full[s]);
                    if (MASK) {
                        if (n >= 2 && !mbar_wait(&m_empty[s], ph, &abort_flag, a.status)) break;
                        mbar_expect_tx(&m_full[s], 2 * kBlockQ);
                        for (int w = 0; w < 2; ++w) tma_load_2d(ms + (2 * s + w) * kBlockQ, &mmap, j0, i0 + w * kTileQ, &m_full[s]);
                    }
                }
                if (n > 0) {
                    const int v = n - 1, s = v & 1;
                    if (v >= 2 && !mbar_wait(&v_empty[s], ((v >> 1) - 1) & 1, &abort_flag, a.status)) break;
                    mbar_expect_tx(&v_full[s], EB * kBlockK);
                    for (int b = 0; b < EB; ++b) tma_load_3d(vs + (s * EB + b) * kBlockK, &vmap, b * 64, h, v * kTileK, &v_full[s]);
                }
            }
        }
    } else if (warp == 1) {
        // the whole warp keeps step, one elected lane issues
        const uint32_t idesc_s = umma_idesc_f16(kTileQ, kTileK);
        const uint32_t idesc_o = umma_idesc_f16(kTileQ, (a.E + 15) & ~15) | (1u << 16);     // V is stored with its columns contiguous
        const uint64_t qd = umma_desc_sw128(qs), kd = umma_desc_sw128(ks), vd = umma_desc_sw128_mn(vs, kBlockK);
        const bool leader = elect_one();
        auto wait = [&](uint64_t* bar, int phase) { return (bool)__all_sync(0xffffffffu, mbar_wait_spin(bar, phase & 1, &abort_flag, a.status)); };
        bool ok = wait(&q_full, 0);
        tc_fence_after();
        for (int n = 0; n <= tiles && ok; ++n) {
            const int s = n & 1, p = s ^ 1;
            if (n < tiles) {
                ok = wait(&k_full[s], n >> 1);
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    if (!ok || (w == 1 && !second)) continue;
                    if (n >= 2) ok = wait(&pv_done[w], n - 2);          // the buffer's last weights have been read
                    if (!ok) continue;
                    tc_fence_after();
                    if (leader) {
                        const uint32_t t = tmem + (uint32_t)w * 256 + 64 * s;
                        const uint64_t bd = kd + (uint64_t)(s * NB * (kBlockK >> 4));
#pragma unroll
                        for (int b = 0; b < NB; ++b)
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                umma_f16(t, qd + (w * NB + b) * (kBlockQ >> 4) + 2 * k, bd + b * (kBlockK >> 4) + 2 * k, idesc_s, (b > 0 || k > 0) ? 1u : 0u);
                        umma_commit(&s_full[w][s]);
                    }
                    __syncwarp();
                }
                if (!ok) break;
                if (leader) umma_commit(&k_empty[s]);
                __syncwarp();
            }
            if (n > 0) {
                ok = wait(&v_full[p], (n - 1) >> 1);
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    if (!ok || (w == 1 && !second)) continue;
                    ok = wait(&p_full[w][p], (n - 1) >> 1);
                    if (!ok) continue;
                    tc_fence_after();
                    if (leader) {
                        const uint32_t t = tmem + (uint32_t)w * 256;
                        const uint64_t bd = vd + (uint64_t)(p * EB * (kBlockK >> 4));
                        const uint32_t more = n > 1 ? 1u : 0u;
#pragma unroll
                        for (int k = 0; k < kTileK / 16; ++k)      // 16 keys are two 1024-byte groups of V, eight columns of P
                            umma_f16_ta(t + 128, t + 64 * p + 8 * k, bd + 128 * k, idesc_o, k > 0 ? 1u : more);
                        umma_commit(&pv_done[w]);
                    }
                    __syncwarp();
                }
                if (!ok) break;
                if (leader) umma_commit(&v_empty[p]);
                __syncwarp();
            }
        }
        if (!ok && leader) {            // given up: let the products in flight end before tensor memory is freed
            umma_commit(&drained);
            for (int i = 0; i < (1 << 20) && !gemvq8::mbar_test_wait(&drained, 0); ++i) {}
        }
        __syncwarp();
    } else if (warp < 6 || second) {
        const int w = warp < 6 ? 0 : 1, quarter = warp & 3;
        const int rw = quarter * 32 + lane, r = w * kTileQ + rw;               // row of the tile, query of the CTA
        const uint32_t t = tmem + (uint32_t)w * 256 + ((uint32_t)(quarter * 32) << 16);
        constexpr float kLog2e = 1.4426950408889634f;
        float sc = a.scale32 ? *a.scale32 : 1.f;
        if (a.scale_q) sc *= __half2float(*a.scale_q);
        if (a.scale_k) sc *= __half2float(*a.scale_k);
        if (!MASK) sc *= kLog2e;                                              // scores in units of log 2; with a mask after the roundings
        const int ocols = (a.E + 31) & ~31;
        float m = -INFINITY, l = 0.f;
        bool ok = true;
        for (int n = 0; n < tiles; ++n) {
            const int b = n & 1;
            uint4 mv[8];
            if (MASK) {
                ok = __all_sync(0xffffffffu, mbar_wait_spin(&m_full[b], (n >> 1) & 1, &abort_flag, a.status));
                if (!ok) break;
                const unsigned char* line = ms + (2 * b + w) * kBlockQ + rw * 128;
#pragma unroll
                for (int c = 0; c < 8; ++c) mv[c] = *reinterpret_cast<const uint4*>(line + ((c ^ (rw & 7)) << 4));
            }
            ok = __all_sync(0xffffffffu, mbar_wait_spin(&s_full[w][b], (n >> 1) & 1, &abort_flag, a.status));
            if (!ok) break;
            tc_fence_after();
            float s[64];
            tmem_ld_32x64(t + 64 * b, s);
            if (MASK) {
                const uint32_t* mw = reinterpret_cast<const uint32_t*>(mv);
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const __half2 z = __hadd2_rn(__floats2half2_rn(s[2 * j] * sc, s[2 * j + 1] * sc), *reinterpret_cast<const __half2*>(&mw[j]));
                    const float2 f = __half22float2(z);
                    s[2 * j] = f.x;
                    s[2 * j + 1] = f.y;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 64; ++j) s[j] *= sc;
            }
            const int left = a.L - n * kTileK;
            if (left < kTileK) {
#pragma unroll
                for (int j = 0; j < 64; ++j)
                    if (j >= left) s[j] = -INFINITY;
            }
            float top4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
            for (int j = 4; j < 64; ++j) top4[j & 3] = fmaxf(top4[j & 3], s[j]);
            constexpr float unit = MASK ? kLog2e : 1.f;
            const float top = fmaxf(fmaxf(top4[0], top4[1]), fmaxf(top4[2], top4[3])) * unit;
            // the maximum that weights are taken against only moves when a score exceeds it by more than 2^8, so that O is rescaled rarely
            const bool move = top > m + 8.f || (m == -INFINITY && top > -INFINITY);
            const float next = move ? top : m;
            const float corr = move ? ex2(m - next) : 1.f;                    // 0 while no key has been seen
            m = next;
            const float z = m == -INFINITY ? 0.f : -m;
            float l4[4] = {l * corr, 0.f, 0.f, 0.f};
            uint32_t pw[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float x = MASK ? ex2(fmaf(s[2 * j], unit, z)) : ex2(s[2 * j] + z), y = MASK ? ex2(fmaf(s[2 * j + 1], unit, z)) : ex2(s[2 * j + 1] + z);
                l4[j & 3] += x + y;
                const __half2 p = __floats2half2_rn(x, y);
                pw[j] = *reinterpret_cast<const uint32_t*>(&p);
            }
            l = (l4[0] + l4[1]) + (l4[2] + l4[3]);
            // O may be rescaled once the product of the tile before has been added.  The last tile always waits for that: a wait for
            // the last product then never looks two completions back.
            const bool any = __any_sync(0xffffffffu, move);
            if (n > 0 && (any || n == tiles - 1)) {
                ok = __all_sync(0xffffffffu, mbar_wait_spin(&pv_done[w], (n - 1) & 1, &abort_flag, a.status));
                if (!ok) break;
                tc_fence_after();
                if (any) {
                    for (int c = 0; c < ocols; c += 32) {
                        float o[32];
                        tmem_ld_32x32(t + 128 + c, o);
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] *= corr;
                        tmem_st_32x32(t + 128 + c, reinterpret_cast<const uint32_t*>(o));
                    }
                }
            }
            tmem_st_32x32(t + 64 * b, pw);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&p_full[w][b]);
                // The mask's piece is given back here, behind the store of weights that depend on every value of it: its loads are over.  Given
                // back right behind the loads, keys of one 16-byte chunk lost their weight in 1 to 5 % of the passes over 199 positions - as if
                // the next piece had come before the last load.  Why is not established (the reads are ordinary ones, the refill is TMA's, and an
                // arrive speaks of accesses of one kind); values that have been used are what this ring and the others rest on.
                if (MASK) mbar_arrive(&m_empty[b]);
            }
        }
        if (ok) {
            ok = __all_sync(0xffffffffu, mbar_wait(&pv_done[w], (tiles - 1) & 1, &abort_flag, a.status));
            tc_fence_after();
            if (ok) {
                const float inv = 1.0f / l;
                __half* out = a.out + ((size_t)(i0 + r) * a.H + h) * a.E;
                for (int c = 0; c < ocols; c += 32) {
                    float o[32];
                    tmem_ld_32x32(t + 128 + c, o);
                    if (r < nq) {
#pragma unroll
                        for (int j = 0; j < 32; j += 8)
                            if (c + j < a.E) {          // E is a multiple of 8
                                __align__(16) __half2 v[4];
#pragma unroll
                                for (int e = 0; e < 4; ++e) v[e] = __floats2half2_rn(o[j + 2 * e] * inv, o[j + 2 * e + 1] * inv);
                                *reinterpret_cast<uint4*>(out + c + j) = *reinterpret_cast<const uint4*>(v);
                            }
                    }
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

// f16, a box of 64 columns x `box_rows` rows (of one head), 128-byte swizzle; what lies beyond the extents reads as zero
bool map_heads(CUtensorMap* map, const HeadRows& t, uint64_t cols, uint64_t heads, uint64_t rows, uint32_t box_rows) {
    gemvq8::EncodeTiledFn fn = gemvq8::encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {cols, heads, rows};
    cuuint64_t strides[2] = {t.head * 2, t.row * 2};
    cuuint32_t box[3] = {64, 1, box_rows};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(t.data), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool map_rows(CUtensorMap* map, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch, uint32_t box_rows) {
    gemvq8::EncodeTiledFn fn = gemvq8::encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {pitch * 2};
    cuuint32_t box[2] = {64, box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr size_t smem_of(int nb, int eb, bool mask) { return 1024 + (size_t)2 * nb * kBlockQ + (size_t)2 * (nb + eb) * kBlockK + (mask ? (size_t)4 * kBlockQ : 0); }

}  // namespace

bool rcu_attention_f16_takes(const rcu_device* dev, const AttentionArgs& a) {
    if (a.T < 2 || a.L < 1 || a.H < 1 || a.H > 0x7fffffff / 128 || a.T > 65535 * kTileQ || a.L > (1 << 30)) return false;
    if (a.D < 8 || a.D > 128 || a.D % 8 || a.E < 8 || a.E > 128 || a.E % 8) return false;
    for (const HeadRows* t : {&a.q, &a.k, &a.v})
        if (t->head % 8 || t->row % 8 || t->head == 0 || t->row == 0) return false;
    return smem_of((a.D + 63) / 64, (a.E + 63) / 64, a.mask != nullptr) + 1024 <= (size_t)dev->smem_optin;
}

rcu_status rcu_attention_f16(rcu_device* dev, const AttentionArgs& a) {
    if (!rcu_attention_f16_takes(dev, a)) return RCU_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(a.q.data) | reinterpret_cast<uintptr_t>(a.k.data) | reinterpret_cast<uintptr_t>(a.v.data) | reinterpret_cast<uintptr_t>(a.out)) & 15)
        return RCU_ERR_UNSUPPORTED;
    const int nb = (a.D + 63) / 64, eb = (a.E + 63) / 64;
    const bool mask = a.mask != nullptr;
    CUtensorMap qm, km, vm, mm;
    // a mask whose rows do not start on 16 bytes is copied with padded rows (the map gives its true width)
    void* padded = nullptr;
    const void* mbase = a.mask;
    uint64_t mpitch = (uint64_t)a.L;
    if (mask && (a.L % 8 || (reinterpret_cast<uintptr_t>(a.mask) & 15))) {
        mpitch = ((uint64_t)a.L + 7) & ~7ull;
        rcu_status st = rcu_alloc(dev, (uint64_t)a.T * mpitch * 2, &padded);
        if (st == RCU_OK) st = rcu_copy2d_pitched(dev, a.mask, padded, a.T, (size_t)a.L * 2, (size_t)a.L * 2, mpitch * 2);
        if (st != RCU_OK) {
            if (padded) rcu_free(dev, padded);
            return st;
        }
        mbase = padded;
    }
    bool maps = map_heads(&qm, a.q, a.D, a.H, a.T, kTileQ) && map_heads(&km, a.k, a.D, a.H, a.L, kTileK) && map_heads(&vm, a.v, a.E, a.H, a.L, kTileK);
    if (mask) maps = maps && map_rows(&mm, mbase, a.L, a.T, mpitch, kTileQ);
    else mm = qm;                     // never read
    if (!maps) {
        if (padded) rcu_free(dev, padded);
        return rcu_fail(dev, RCU_ERR_CUDA, "attention: cuTensorMapEncodeTiled failed (T=%d L=%d H=%d D=%d)", a.T, a.L, a.H, a.D);
    }
    // two tiles take turns on the tensor cores and in the softmax; where they leave most SMs idle one is better (6 heads of 501 positions, 12 CTAs: 14.7 us, 24 with a tile each: 11.2)
    const int per = 2 * a.H * ((a.T + 2 * kTileQ - 1) / (2 * kTileQ)) <= dev->sm_count ? kTileQ : 2 * kTileQ;
    const Args t{(__half*)a.out, a.H, a.T, a.L, a.E, per, a.scale32[0], a.scale16[0], a.scale16[1], dev->d_status};
    const dim3 grid(a.H, (a.T + per - 1) / per);
    const size_t smem = smem_of(nb, eb, mask);
    void (*kern)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, Args);
#define RCU_ATT(NB_, EB_) kern = mask ? attention_kernel<NB_, EB_, true> : attention_kernel<NB_, EB_, false>
    if (nb == 1 && eb == 1) RCU_ATT(1, 1);
    else if (nb == 1) RCU_ATT(1, 2);
    else if (eb == 1) RCU_ATT(2, 1);
    else RCU_ATT(2, 2);
#undef RCU_ATT
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = rcu_launch(dev, kern, grid, kThreadsA, smem, qm, km, vm, mm, t);
    if (padded) rcu_free(dev, padded);          // the pool reuses blocks in stream order
    if (e != cudaSuccess) return rcu_fail(dev, RCU_ERR_CUDA, "attention: %s", cudaGetErrorString(e));
    RCU_LAUNCH_CHECK(dev);
    return RCU_OK;
}
