// Prefill GEMM on CTA pairs (tcgen05 cta_group::2), Linear convention:
//   out[M, N] = X[M, K] . W[N, K]^T (+ bias),  X, W and out f16, f32 accumulation in tensor memory.
//
// Same contract as gemm_tc_kernel (ops/matmul/gemm.rs:462-746 is what it stands in for); used for
// f16 weights when the problem has at least a few 256 x 256 tiles.  A 128 x 256 x 16 MMA of one CTA
// reads 12 KiB of operands from shared memory in the 128 cycles it takes, and TMA writes the same
// amount: together more than the 128 bytes per cycle an SM's shared memory moves, which is what held
// the one-CTA kernel near two thirds of the tensor rate.  Here two CTAs of a cluster compute one
// 256 x 256 tile: each holds 128 token rows of X and 128 of the tile's 256 weight rows, the pair's
// tensor cores exchange the weight halves, and every CTA reads and writes 8 KiB per MMA.
//
//   warp 0 (one lane)  TMA producer: its CTA's 128 x 64 X tile and 128 x 64 W tile per stage, completion
//                      counted on the LEADER CTA's `full` barrier (the leader expects both CTAs' bytes);
//   warp 1 (leader CTA only; one elected lane)  issues four tcgen05.mma.cta_group::2 per stage and commits them
//                      to the stage's `empty` barrier of both CTAs, and at the end of a tile to both CTAs'
//                      `acc_full` barrier;
//   warps 2-9          epilogue of the CTA's own 128 rows, two warps per tensor-memory lane quarter: tcgen05.ld, 32 x 32
//                      pieces turned around in shared memory, bias, activation, residual, whole lines to memory; then one
//                      arrival per warp on the leader's `acc_empty` barrier.
// Quantised weights (Q8_0H, Q4_KH; WK): the W tile's place is filled by eight further warps, which convert the codes of their CTA's 128
// rows with the CPU dequantiser's arithmetic and write the swizzled tile; the leader's `full` barrier counts their warps beside the TMA's bytes of X.
//   warps 10-17        convert, in four teams of two, each every fourth step of 64 of K: what a step costs a warp is a chain - waits, conversion,
//                      fence, arrival: 1200 cycles when eight warps shared it - and a step's MMAs take 512;
//   warp 18            brings the codes: TMA, a ring of their own;
//   warp 19            the scales: plain loads, sixteen bytes a row for four steps (requested by the converting warps themselves, codes and
//                      scales took 2000 cycles a step: 1500 sectors in flight per SM).
// The converting warps arrive in CTA scope: the tensor cores read behind a proxy fence; arriving in cluster scope waited 0.65 us a step for L2.
// 512 x 8192 x 3072 Q4_KH: 35.1 us with the conversion in front of it -> 33.7; 512 x 9216 x 3072 Q8_0H: 37.3 -> 31.4 (pair_converts in gemm_tc.cu has more).
// What bounds it: the chain of hand-overs - a step takes some 1000 cycles with the tensor pipe 40 to 45 % busy, issue slots 33 % - and with Q8_0 the codes' and the
// converted tile's way through shared memory as well (52 % of its wavefronts are the converting warps').
//
// The kernel is persistent: a pair walks over tiles pair, pair + n_pairs, ...; the accumulator is
// double-buffered (2 x 256 of the 512 tensor-memory columns), so the epilogue of tile i overlaps the
// MMAs of tile i + 1.  Tiles that share a weight tile run on neighbouring pairs at the same time (the
// activations, M x K, stay in L2).
//
// Every wait is bounded (mbar_wait); a wait that gives up raises RCU_DEVFLAG_TIMEOUT and ends the
// CTA's other waits through a flag in shared memory.  Both CTAs meet at a cluster barrier before tensor
// memory is freed, so neither touches the other's shared memory after it has exited.
#include <cuda.h>

#include <type_traits>

#include "dequant.cuh"
#include "lm_math.cuh"
#include "tc_common.cuh"

namespace {

using namespace tc;

constexpr int kStages2 = 6;
constexpr int kTileN2 = 256;                       // weight rows per pair tile (128 per CTA)
constexpr int kStageBytes2 = 2 * TM * TK * 2;      // 128 x 64 f16 of X + 128 x 64 f16 of W = 32 KiB
constexpr int kEpilogueWarps = 8;                  // two per tensor-memory lane quarter, half of the columns each
constexpr int kThreads2 = 64 + kEpilogueWarps * 32;
constexpr int kAccCols = 256;                      // f32 accumulator columns per buffer
constexpr int kConvWarps = 8;                      // converting warps of a CTA (quantised weights)
constexpr int kTeams = 4, kTeamWarps = kConvWarps / kTeams, kFeedWarps = 2;
constexpr int kGroup = 4;                          // steps whose scales travel together: 256 of K
constexpr int kScaleSlots = 2;                     // groups of scales in flight
constexpr int stages2(int wk) { return wk == WK_F16 ? kStages2 : wk == WK_Q8 ? 4 : 5; }
constexpr int raw_slots(int wk) { return wk == WK_F16 ? 0 : 4; }                // steps of codes in flight
constexpr int free_slots(int wk) { return wk == WK_Q4K ? 8 : 0; }               // stages that are handed on (RawRings); 0: the teams wait for them themselves
constexpr int raw_row(int wk) { return wk == WK_Q8 ? TK : TK / 2; }             // bytes of a row's codes in a step
constexpr int scale_row(int wk) { return wk == WK_Q8 ? 16 : 32; }               // of its scales in a group: eight f16; eight multipliers and minima
constexpr int raw_bytes(int wk) { return wk == WK_F16 ? 0 : TM * (raw_slots(wk) * raw_row(wk) + kScaleSlots * scale_row(wk)); }
constexpr int threads2(int wk) { return kThreads2 + (wk == WK_F16 ? 0 : (kConvWarps + kFeedWarps) * 32); }
constexpr size_t smem2(int wk) { return 1024 + (size_t)stages2(wk) * kStageBytes2 + raw_bytes(wk) + 512; }

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// address of `local` (a shared-memory address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// the same in CTA scope: for the async proxy's reads (behind fence.proxy.async), which need no fence across the cluster - that one waits for
// the thread's writes to reach L2
__device__ __forceinline__ void mbar_arrive_peer(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// TMA tile load whose completion is counted on a barrier that may live in the peer CTA
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(bar_cluster_addr)
        : "memory");
}
__device__ __forceinline__ void umma2_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrive on the barrier at this shared-memory offset in both CTAs of the pair once every MMA issued so far is done
__device__ __forceinline__ void umma2_commit_both(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}

// What the converting warps of a CTA work from.  A barrier's parity tells a use of a slot from the one before it, not from one further back, and
// neither loads nor commits on different barriers need arrive in the order that they were asked for.  So whoever waits for a use of a slot must be who waited
// for the use before it.  A team has every fourth step (K is whole groups: a tile does not shift the teams), so the ring of codes is a multiple of
// four slots.  (Of six slots a team met every second fill only, whose parity it had seen already: a load that the one behind it overtook was not waited
// for.)  So are Q8_0's stages.  Q4_K's five are not - with four 512 x 8192 x 3072 takes 39.0 us, not 33.4 - so the warp that brings the activations, which waits for
// every use of every stage, hands each on through a ring of eight: more than it can be ahead.
struct RawRings {
    unsigned char *codes, *scales;              // [raw_slots][128][raw_row], [kScaleSlots][128][scale_row]
    uint64_t *full, *empty, *scale_full, *scale_empty, *stage_free;
};
// The first row of W that this CTA has of tile t
template <bool GLU> __device__ __forceinline__ int tile_row(int t, int tiles_m, uint32_t rank, int N) {
    return GLU ? (t / tiles_m) * (kTileN2 / 2) + (int)rank * N : (t / tiles_m) * kTileN2 + (int)rank * (kTileN2 / 2);
}

template <int WK, bool GLU>
__device__ __forceinline__ void feed_codes(const CUtensorMap* wmap, const RawRings& raw, uint32_t rank, int pair, int n_pairs, int n_tiles, int tiles_m, int N, int nk,
                                           volatile int* abort_flag, int* status) {
    constexpr int SLOTS = raw_slots(WK);
    if ((threadIdx.x & 31) != 0) return;
    int it = 0, rs = 0, phase = 1;            // a fresh barrier's odd phase counts as done
    for (int t = pair; t < n_tiles; t += n_pairs) {
        const int row = tile_row<GLU>(t, tiles_m, rank, N);
        for (int k = 0; k < nk; ++k, ++it) {
            if (!mbar_wait(&raw.empty[rs], (unsigned)phase, abort_flag, status)) {
                // given up: the codes in flight get another chance to land before the CTA leaves
                for (int i = 1; i <= min(it, SLOTS); ++i)
                    for (int n = 0; n < (1 << 16) && !gemvq8::mbar_test_wait(&raw.full[(it - i) % SLOTS], ((it - i) / SLOTS) & 1); ++n) {}
                return;
            }
            mbar_expect_tx(&raw.full[rs], TM * raw_row(WK));
            tma_load_2d(raw.codes + rs * TM * raw_row(WK), wmap, k * raw_row(WK), row, &raw.full[rs]);
            if (++rs == SLOTS) { rs = 0; phase ^= 1; }
        }
    }
}

// Q8_0: a row's block scales as they are.  Q4_K: of each sub-block fp(scale d) and -fp(min dmin), small integers times f16, rounded once
// (quantized.rs:158-204).  Rows beyond the matrix get zeros.
template <int WK, bool GLU>
__device__ __forceinline__ void feed_scales(const QuantArgs& qa, const RawRings& raw, uint32_t rank, int pair, int n_pairs, int n_tiles, int tiles_m, int rows, int N, int K,
                                            volatile int* abort_flag, int* status) {
    using namespace rcu_dequant;
    const int lane = threadIdx.x & 31, groups = K / (kGroup * TK);
    uint4 next[4];
    auto request = [&](int t, int group) {
        const int n0 = tile_row<GLU>(t, tiles_m, rank, N);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = n0 + 32 * i + lane;
            next[i] = make_uint4(0u, 0u, 0u, 0u);
            if (t >= n_tiles || row >= rows) continue;
            if (WK == WK_Q8) {
                next[i] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(qa.scales) + (size_t)row * (K >> 5) + group * 8));
            } else {
                const size_t block = (size_t)row * (K >> 8) + group;
                const uint32_t* g = reinterpret_cast<const uint32_t*>(qa.scales) + block * 3;
                const uint32_t d = __ldg(reinterpret_cast<const unsigned short*>(qa.d) + block), m = __ldg(reinterpret_cast<const unsigned short*>(qa.dmin) + block);
                next[i] = make_uint4(__ldg(g), __ldg(g + 1), __ldg(g + 2), d | m << 16);
            }
        }
    };
    request(pair, 0);
    int gs = 0, phase = 1;
    for (int t = pair; t < n_tiles; t += n_pairs) {
        for (int g = 0; g < groups; ++g) {
            const uint4 now[4] = {next[0], next[1], next[2], next[3]};
            const bool end = g + 1 == groups;
            request(end ? t + n_pairs : t, end ? 0 : g + 1);
            if (!__all_sync(0xffffffffu, mbar_wait(&raw.scale_empty[gs], (unsigned)phase, abort_flag, status))) return;
            uint4* slot = reinterpret_cast<uint4*>(raw.scales + gs * TM * scale_row(WK));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = 32 * i + lane;
                if (WK == WK_Q8) {
                    slot[r] = now[i];
                } else {
                    // four sub-blocks' scales or minima in a word's bytes
                    const uint32_t six[4] = {now[i].x & 0x3F3F3F3Fu, (now[i].z & 0x0F0F0F0Fu) | ((now[i].x >> 2) & 0x30303030u), now[i].y & 0x3F3F3F3Fu,
                                             ((now[i].z >> 4) & 0x0F0F0F0Fu) | ((now[i].y >> 2) & 0x30303030u)};
                    const __half2 k1024 = __float2half2_rn(1024.0f), d2 = __low2half2(as_h2(now[i].w)), min2 = __high2half2(as_h2(now[i].w));
                    uint32_t mn[8];
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const uint32_t sel = j & 2 ? 0x4342u : 0x4140u;
                        const uint32_t mul = as_u32(__hmul2_rn(__hsub2_rn(as_h2(prmt(six[j >> 2], 0x64646464u, sel)), k1024), d2));
                        const uint32_t neg = as_u32(__hneg2(__hmul2_rn(__hsub2_rn(as_h2(prmt(six[2 + (j >> 2)], 0x64646464u, sel)), k1024), min2)));
                        mn[j] = prmt(mul, neg, 0x5410u);
                        mn[j + 1] = prmt(mul, neg, 0x7632u);
                    }
                    slot[2 * r] = make_uint4(mn[0], mn[1], mn[2], mn[3]);
                    slot[2 * r + 1] = make_uint4(mn[4], mn[5], mn[6], mn[7]);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw.scale_full[gs]);
            if (++gs == kScaleSlots) { gs = 0; phase ^= 1; }
        }
    }
}

// The converting warps: 64 rows of every fourth step of the W tiles that the pair works on.
//   Q8_0: four lanes per row, sixteen codes of one block each; lanes 0-7 of a store write eight different chunks.
//   Q4_K: two lanes per row, sixteen bytes each: low nibbles belong to the step's first sub-block, high ones to its second.  Rows 2 and 3 of
//   every four store the second one first: eight lanes then write eight different chunks.
template <int WK>
__device__ __forceinline__ void convert_tiles(const RawRings& raw, unsigned char* smem, uint64_t* full, uint64_t* empty, int steps, volatile int* abort_flag, int* status) {
    using namespace rcu_dequant;
    constexpr int SLOTS = raw_slots(WK), FREE = free_slots(WK), S = stages2(WK);
    static_assert(kTeams == kGroup, "a team has one step of every group: its index is the step's place there");
    static_assert(SLOTS % kTeams == 0 && (FREE ? FREE % kTeams == 0 && FREE > S : S % kTeams == 0), "a slot belongs to one team");
    constexpr int PER_ROW = WK == WK_Q8 ? 4 : 2, TASKS = TM / kTeamWarps * PER_ROW / 32, ROWS = 32 / PER_ROW;      // lanes per row; rows of a lane, so far apart
    const int lane = threadIdx.x & 31, cw = (threadIdx.x - kThreads2) >> 5, team = cw / kTeamWarps;
    const int r0 = cw % kTeamWarps * (TM / kTeamWarps) + lane / PER_ROW, part = lane % PER_ROW;
    const uint32_t full_leader = map_to_cta(smem_u32(full), 0);
    auto wait = [&](uint64_t* bar, int parity) { return (bool)__all_sync(0xffffffffu, mbar_wait(bar, (unsigned)parity, abort_flag, status)); };
    int gs = 0, scale_phase = 0;
    for (int it = team; it < steps; it += kTeams) {
        const int s = it % S, rs = it % SLOTS;
        if (!wait(&raw.scale_full[gs], scale_phase) || !wait(&raw.full[rs], (it / SLOTS) & 1)) return;
        const unsigned char *codes = raw.codes + rs * TM * raw_row(WK), *scales = raw.scales + gs * TM * scale_row(WK);
        uint4 q[TASKS], o[TASKS][WK == WK_Q8 ? 2 : 4];
        uint2 sc[TASKS];
#pragma unroll
        for (int i = 0; i < TASKS; ++i) {
            const int r = r0 + ROWS * i;
            q[i] = *reinterpret_cast<const uint4*>(codes + r * raw_row(WK) + part * 16);
            if (WK == WK_Q8) sc[i].x = *reinterpret_cast<const unsigned short*>(scales + r * 16 + 4 * team + 2 * (part >> 1));
            else sc[i] = *reinterpret_cast<const uint2*>(scales + r * 32 + 8 * team);
        }
#pragma unroll
        for (int i = 0; i < TASKS; ++i) {
            if (WK == WK_Q8) {
                const __half2 m = __half2half2(__ushort_as_half((unsigned short)sc[i].x));
                o[i][0] = dequant8_q8(q[i].x, q[i].y, m);
                o[i][1] = dequant8_q8(q[i].z, q[i].w, m);
            } else {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int h = x ^ ((r0 >> 1) & 1);
                    const __half2 mn = as_h2(h ? sc[i].y : sc[i].x), mul = __low2half2(mn), neg = __high2half2(mn);
                    o[i][2 * x] = dequant8_q4(q[i].x >> (4 * h), q[i].y >> (4 * h), mul, neg);
                    o[i][(WK == WK_Q8 ? 0 : 2 * x) + 1] = dequant8_q4(q[i].z >> (4 * h), q[i].w >> (4 * h), mul, neg);
                }
            }
        }
        __syncwarp();                         // every lane has its codes and scales
        if (lane == 0) {
            mbar_arrive(&raw.empty[rs]);
            mbar_arrive(&raw.scale_empty[gs]);
        }
        if (++gs == kScaleSlots) { gs = 0; scale_phase ^= 1; }
        if constexpr (FREE > 0) {
            if (!wait(&raw.stage_free[it % FREE], (it / FREE) & 1)) return;
        } else {
            if (!wait(&empty[s], (it / S + 1) & 1)) return;     // a fresh barrier's odd phase counts as done
        }
        unsigned char* tile = smem + s * kStageBytes2 + TM * TK * 2;
#pragma unroll
        for (int i = 0; i < TASKS; ++i) {
            const int r = r0 + ROWS * i;
            unsigned char* line = tile + r * 128;
#pragma unroll
            for (int x = 0; x < (WK == WK_Q8 ? 2 : 4); ++x) {
                const int chunk = WK == WK_Q8 ? 2 * part + x : 4 * ((x >> 1) ^ ((r0 >> 1) & 1)) + 2 * part + (x & 1);
                *reinterpret_cast<uint4*>(line + ((chunk ^ (r & 7)) << 4)) = o[i][x];
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // plain stores, read by the tensor cores
        __syncwarp();
        if (lane == 0) mbar_arrive_peer(full_leader + (uint32_t)(s * 8));
    }
}

// glu_value: a gate and an up value as the graph's own kernels have them - f16: half_chains.cu (silu rounded before the product),
// bf16: glu_kernel of stream_ops.cu
template <class Out> __device__ __forceinline__ float glu_value(int act, float gate, float up) {
    gate = rnd<Out>(gate);
    up = rnd<Out>(up);
    if constexpr (std::is_same<Out, __half>::value) return up * rnd<Out>(chain_act(act, gate));
    else return (act == RCU_GELU ? lm::gelu_tanh(gate) : lm::silu(gate)) * up;
}

// GLU: W holds N gate rows, then N up rows; a tile's first CTA brings 128 gate rows, the second their up rows, and the output tile is 128
// columns wide.  Written separately, the product and its gate cost 55 MB of traffic more at 1000 x 2 x 8192 (12.9 us of the kernel that read
// it), 185 MB at 4096 x 2 x 5632 (33.9 us).
template <class Out, int MODE, bool GLU, int WK>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(threads2(WK), 1)
gemm_tc2_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const GemmEpilogue<Out, MODE> epi,
                Out* out, int M, int N, int K, int tiles_m, int n_tiles, int* status, uint32_t idesc, int glu_act, const QuantArgs qa, bool lead) {
    constexpr int STAGES = stages2(WK), RAW = raw_bytes(WK), SLOTS = raw_slots(WK), FREE = free_slots(WK);
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * kStageBytes2 + RAW);   // leader's are the ones in use
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;        // [2]
    uint64_t* acc_empty = acc_full + 2;           // [2], leader's in use
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint64_t* raw_bars = reinterpret_cast<uint64_t*>(tmem_slot + 2);
    const RawRings raw{smem + STAGES * kStageBytes2, smem + STAGES * kStageBytes2 + SLOTS * TM * raw_row(WK), raw_bars, raw_bars + SLOTS,
                       raw_bars + 2 * SLOTS, raw_bars + 2 * SLOTS + kScaleSlots, raw_bars + 2 * SLOTS + 2 * kScaleSlots};

    __shared__ float4 turn[kEpilogueWarps][kTurnQuads];      // one piece of an accumulator per epilogue warp
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();                 // 0 = leader
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int nk = (K + TK - 1) / TK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], WK == WK_F16 ? 1 : 1 + 2 * kTeamWarps);      // the TMA's, a team's warps of either CTA
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * kEpilogueWarps);       // both CTAs'
        }
        if (WK != WK_F16) {
            for (int i = 0; i < SLOTS; ++i) {
                mbar_init(&raw.full[i], 1);
                mbar_init(&raw.empty[i], kTeamWarps);
            }
            for (int i = 0; i < kScaleSlots; ++i) {
                mbar_init(&raw.scale_full[i], 1);
                mbar_init(&raw.scale_empty[i], kConvWarps);
            }
            for (int i = 0; i < FREE; ++i) mbar_init(&raw.stage_free[i], 1);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(2 * kAccCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    cluster_sync_all();            // barriers of both CTAs initialised before anyone signals them
    tc_fence_after();
    rcu_kernel_entry_wait_only();  // nothing before this touches global memory: the set-up overlaps the kernel before
    if (lead) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");      // a conversion for the next product runs beside this one
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int t = pair; t < n_tiles && ok; t += n_pairs) {
                const int m0 = (t % tiles_m) * 2 * TM + (int)rank * TM;
                const int n0 = GLU ? (t / tiles_m) * (kTileN2 / 2) + (int)rank * N : (t / tiles_m) * kTileN2 + (int)rank * (kTileN2 / 2);
                for (int k = 0; k < nk; ++k, ++it) {
                    const int s = it % STAGES;
                    if (it >= STAGES && !mbar_wait(&empty[s], ((it / STAGES) - 1) & 1, abort_flag, status)) { ok = false; break; }
                    if constexpr (FREE > 0) mbar_arrive(&raw.stage_free[it % FREE]);
                    unsigned char* st = smem + s * kStageBytes2;
                    if (rank == 0) mbar_expect_tx(&full[s], WK == WK_F16 ? 2 * kStageBytes2 : kStageBytes2);      // both CTAs' bytes
                    const uint32_t bar = map_to_cta(smem_u32(&full[s]), 0);
                    tma_load_2d_pair(st, &xmap, k * TK, m0, bar);
                    if (WK == WK_F16) tma_load_2d_pair(st + TM * TK * 2, &wmap, k * TK, n0, bar);
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {               // the whole warp keeps step, one elected lane issues
            const bool leader = elect_one();
            const uint64_t desc0 = umma_desc_sw128(smem);
            int s = 0, phase = 0, i = 0;
            bool ok = true;
            for (int t = pair; t < n_tiles && ok; t += n_pairs, ++i) {
                const int b = i & 1;
                if (i >= 2) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[b], ((i >> 1) - 1) & 1, abort_flag, status));
                    if (!ok) break;
                    tc_fence_after();
                }
                const uint32_t acc = tmem_base + (uint32_t)(b * kAccCols);
                for (int k = 0; k < nk; ++k) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&full[s], phase, abort_flag, status));
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) {
                        const uint64_t adesc = desc0 + (uint64_t)(s * (kStageBytes2 >> 4)), bdesc = adesc + (TM * TK * 2 >> 4);
#pragma unroll
                        for (int kk = 0; kk < TK / 16; ++kk) umma2_f16(acc, adesc + 2 * kk, bdesc + 2 * kk, idesc, (k > 0 || kk > 0) ? 1u : 0u);
                        umma2_commit_both(&empty[s]);
                    }
                    __syncwarp();
                    if (++s == STAGES) { s = 0; phase ^= 1; }
                }
                if (leader) umma2_commit_both(&acc_full[b]);      // also after an abort, so that the epilogues end
                __syncwarp();
            }
        }
    } else if (WK != WK_F16 && warp == 2 + kEpilogueWarps + kConvWarps) {
        if constexpr (WK != WK_F16) feed_codes<WK, GLU>(&wmap, raw, rank, pair, n_pairs, n_tiles, tiles_m, N, nk, abort_flag, status);
    } else if (WK != WK_F16 && warp == 3 + kEpilogueWarps + kConvWarps) {
        feed_scales<WK, GLU>(qa, raw, rank, pair, n_pairs, n_tiles, tiles_m, GLU ? 2 * N : N, N, K, abort_flag, status);
    } else if (WK != WK_F16 && warp >= 2 + kEpilogueWarps) {
        if constexpr (WK != WK_F16) convert_tiles<WK>(raw, smem, full, empty, pair < n_tiles ? (n_tiles - pair + n_pairs - 1) / n_pairs * nk : 0, abort_flag, status);
    } else {
        // epilogue warps 2..9: tensor-memory lane quarter = warp index modulo 4
        const int q = warp & 3, c0 = (warp - 2) / 4 * (kTileN2 / 2);
        const uint32_t acc_empty_leader0 = map_to_cta(smem_u32(&acc_empty[0]), 0);
        int i = 0;
        bool ok = true;
        for (int t = pair; t < n_tiles && ok; t += n_pairs, ++i) {
            const int b = i & 1;
            ok = mbar_wait(&acc_full[b], (i >> 1) & 1, abort_flag, status);
            if (!ok) break;
            tc_fence_after();
            const int row0 = (t % tiles_m) * 2 * TM + (int)rank * TM + q * 32;
            const int n0 = (t / tiles_m) * (GLU ? kTileN2 / 2 : kTileN2);
            float4* mine = turn[warp - 2];
            const int r = lane >> 3, quad = lane & 7;
            if constexpr (GLU) {
#pragma unroll 1
                for (int c = c0 / 2; c < c0 / 2 + kTileN2 / 4; c += 32) {
                    const int col = n0 + c + quad * 4;
                    const uint32_t at = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * kAccCols + c);
                    turn_piece8(
                        mine,
                        [&](int c8, float* v) {
                            float u[8];
                            tmem_ld_32x8(at + 8 * c8, v);
                            tmem_ld_32x8(at + kTileN2 / 2 + 8 * c8, u);
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[e] = glu_value<Out>(glu_act, v[e], u[e]);
                        },
                        [&](int i, int piece_row, const float4& x) {
                            const int row = row0 + piece_row;
                            if (col >= N || row >= M) return;
                            typename GemmEpilogue<Out, MODE>::Quad o;
                            o.v[0] = from_f32<Out>(x.x);
                            o.v[1] = from_f32<Out>(x.y);
                            o.v[2] = from_f32<Out>(x.z);
                            o.v[3] = from_f32<Out>(x.w);
                            *reinterpret_cast<decltype(o)*>(out + (size_t)row * N + col) = o;
                        });
                }
            } else {
#pragma unroll 1
            for (int c = c0; c < c0 + kTileN2 / 2; c += 32) {
                const int col = n0 + c + quad * 4;
                const bool in = col < N;
                const float4 bias = in ? epi.bias4(col, N) : make_float4(0.f, 0.f, 0.f, 0.f);
                typename GemmEpilogue<Out, MODE>::Resid resid[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int row = row0 + 4 * i + r;
                    resid[i] = epi.resid4((size_t)row * N + col, in && row < M);
                }
                const uint32_t at = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * kAccCols + c);
                auto put = [&](int i, int piece_row, const float4& x) {
                    const int row = row0 + piece_row;
                    if (in && row < M) epi.store4(out, (size_t)row * N + col, x, bias, resid[i], col, N);
                };
                if constexpr (MODE == EPI_ACT) {
                    turn_piece8(
                        mine,
                        [&](int c8, float* v) {
                            tmem_ld_32x8(at + 8 * c8, v);
                            epi.finish8(v, n0 + c + 8 * c8, N);
                        },
                        put);
                } else {
                    float v[32];
                    tmem_ld_32x32(at, v);
                    turn_piece(mine, v, put);
                }
            }
            }
            // this warp has read its part of the buffer: tell the leader's MMA thread
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(acc_empty_leader0 + (uint32_t)(b * 8));
        }
    }
    tc_fence_before();
    cluster_sync_all();            // the peer may still be signalling barriers in this CTA's shared memory
    tc_fence_after();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(2 * kAccCols) : "memory");
    }
}

bool make_map_f16_sw128_rows(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K, uint32_t box_rows, uint64_t pitch, bool bf16) {
    gemvq8::EncodeTiledFn fn = gemvq8::encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {K, rows};
    cuuint64_t strides[1] = {pitch * 2};
    cuuint32_t box[2] = {(cuuint32_t)TK, box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// RCU_GEMM_PAIR=0 in the environment turns the CTA-pair kernel off
bool rcu_gemm_tc2_on() {
    static const int mode = [] { const char* e = getenv("RCU_GEMM_PAIR"); return e ? atoi(e) : 1; }();
    return mode != 0;
}
// f16 x f16 problems with at least a quarter as many 256 x 256 tiles as SMs take the CTA-pair kernel
bool rcu_gemm_tc2_eligible(rcu_device* dev, uint64_t M, uint64_t N, uint64_t K) {
    if (!rcu_gemm_tc2_on()) return false;
    if (M < 256 || N < 256 || K < 64 || K % 8 != 0) return false;
    const uint64_t tiles = ((M + 255) / 256) * ((N + 255) / 256);
    return tiles >= (uint64_t)dev->sm_count / 4;
}

namespace {
// `N`: rows of W; with a gate the output has half as many columns
template <class Out, int MODE = EPI_PLAIN, bool GLU = false, int WK = WK_F16>
rcu_status launch_pair(rcu_device* dev, const CUtensorMap& xmap, const CUtensorMap& wmap, const GemmEpilogue<Out, MODE>& epi, void* y, uint64_t M, uint64_t N,
                       uint64_t K, const TcLinear& t) {
    const int tiles_m = (int)((M + 255) / 256), tiles_n = (int)((N + 255) / 256);      // a tile of gates takes 256 rows of W too
    const int n_tiles = tiles_m * tiles_n;
    const int n_pairs = std::min(n_tiles, dev->sm_count / 2);
    rcu_device::NextConversion* next = dev->next_conversion;
    constexpr size_t smem = smem2(WK);
    auto kern = gemm_tc2_kernel<Out, MODE, GLU, WK>;
    RCU_CUDA(dev, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    RCU_CUDA(dev, rcu_launch(dev, kern, 2 * n_pairs, threads2(WK), smem, xmap, wmap, epi, (Out*)y, (int)M, (int)(GLU ? N / 2 : N), (int)K, tiles_m, n_tiles, dev->d_status,
                             umma_idesc_f16(2 * TM, kTileN2, t.bf16), t.glu, t.quant, next != nullptr));
    RCU_LAUNCH_CHECK(dev);
    if (next) next->started = rcu_dequantize_beside(dev, *next) == RCU_OK;
    return RCU_OK;
}
}  // namespace

rcu_status rcu_gemm_tc2_launch(rcu_device* dev, const void* w, const void* x, const void* bias, void* y, uint64_t M, uint64_t N, uint64_t K,
                               const TcLinear& t) {
    CUtensorMap xmap, wmap;
    if (!make_map_f16_sw128_rows(&xmap, x, M, K, TM, t.x_pitch ? t.x_pitch : K, t.bf16) ||
        (t.wk == WK_F16 && !make_map_f16_sw128_rows(&wmap, w, N, K, kTileN2 / 2, K, t.bf16)))
        return rcu_fail(dev, RCU_ERR_CUDA, "gemm_tc2: cuTensorMapEncodeTiled failed (M=%llu N=%llu K=%llu)", (unsigned long long)M,
                        (unsigned long long)N, (unsigned long long)K);
    if (t.wk != WK_F16 && !gemvq8::make_map_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, t.quant.codes, N, t.wk == WK_Q8 ? K : K / 2, raw_row(t.wk), kTileN2 / 2))
        return rcu_fail(dev, RCU_ERR_CUDA, "gemm_tc2: cuTensorMapEncodeTiled failed (codes, N=%llu K=%llu)", (unsigned long long)N, (unsigned long long)K);
#define RCU_PAIR(OUT_, MODE_, GLU_, ...) launch_pair<OUT_, MODE_, GLU_>(dev, xmap, wmap, GemmEpilogue<OUT_, MODE_>{(const OUT_*)bias, __VA_ARGS__}, y, M, N, K, t)
#define RCU_PAIR_H(MODE_, GLU_, ...)                                                                                                                                             \
    (t.wk == WK_Q8    ? launch_pair<__half, MODE_, GLU_, WK_Q8>(dev, xmap, wmap, GemmEpilogue<__half, MODE_>{(const __half*)bias, __VA_ARGS__}, y, M, N, K, t)                 \
     : t.wk == WK_Q4K ? launch_pair<__half, MODE_, GLU_, WK_Q4K>(dev, xmap, wmap, GemmEpilogue<__half, MODE_>{(const __half*)bias, __VA_ARGS__}, y, M, N, K, t)                \
                      : RCU_PAIR(__half, MODE_, GLU_, __VA_ARGS__))
    if (t.glu >= 0) return t.bf16 ? RCU_PAIR(__nv_bfloat16, EPI_PLAIN, true, nullptr, 1.f, {}) : RCU_PAIR_H(EPI_PLAIN, true, nullptr, 1.f, {});
    if (t.out_dt == RCU_F32) return RCU_PAIR(float, EPI_PLAIN, false, t.resid, t.alpha, t.act);
    if (t.out_dt == RCU_BF16) return RCU_PAIR(__nv_bfloat16, EPI_PLAIN, false, nullptr, 1.f, t.act);
    if (t.chain_op >= 0) return RCU_PAIR_H(EPI_ACT, false, nullptr, 1.f, {}, t.bias32, nullptr, t.chain_op);
    if (t.chained()) return RCU_PAIR_H(EPI_RESID, false, nullptr, 1.f, {}, t.bias32, (const __half*)t.resid16, -1);
    if (N & 3) return RCU_PAIR_H(EPI_RAGGED, false, nullptr, 1.f, t.act);
    return RCU_PAIR_H(EPI_PLAIN, false, nullptr, 1.f, t.act);
#undef RCU_PAIR
#undef RCU_PAIR_H
}
