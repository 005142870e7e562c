// Linear over a few token rows (a short prompt, a speculative batch), ratchet's convention:
//   out[M, N] = X[M, K] . W[N, K]^T (+ bias),  X and out f16, W f16, Q8_0H, Q8_0F or Q4_KH, f32 accumulation.
//
// Stands in for ratchet-core's `gemm` (ops/matmul/gemm.rs:462-746) where a product is still the stream of its weights: up to a few
// dozen rows the tensor work is hidden behind the bytes of W, so what counts is that W arrives at memory speed and is unpacked once.
// The weights go from global memory into registers, become f16 there and are the A operand (16 rows x 16 k) of mma.sync; eight
// token rows are the B operand.  The order of k inside a chunk is chosen for the loads: a lane's elements of a row are consecutive, so
// that the quad's four lanes read whole lines of W and a lane unpacks with one or two scales, and the same elements of the token rows
// come from L1 / L2.  (A first form read 32 bytes of a row at a time: 48 us instead of 23 for two rows, 32001 x 3072 Q8_0H.)  The warps
// of a CTA take turns at the chunks of the same rows and add up through shared memory.  No operand passes through shared memory, so nothing but registers limits how many loads are in flight.
//
// Q8_0F keeps its 32-bit block scales out of the f16 product: the codes (exact in f16) of one 32-element block are multiplied with
// the tokens in an accumulator of their own, which enters the sum through an f32 fma with the block's scale.  This form serves any
// number of token rows (blockIdx.y).
//
// Measured on B200 (us, K = 3072, 2 / 16 / 32 rows, weights that rotate through more than L2, from a CUDA graph; before: the SIMT kernel, which
// unpacks every weight anew for each 64-row tile and multiplies on the FMA pipe; 32 rows of Q8_0H, Q4_KH and f16 at N = 32001 are not this kernel's):
//             N = 3072                              N = 9216                               N = 32001
//   Q8_0H   213 / 209 / 13 -> 5.3 / 6.6 / 8.9    253 / 251 / 20 ->  8.6 / 13 / 17     570 / 581 / 593 -> 25 / 39 /  -
//   Q8_0F   239 / 242 / 240 -> 8.5 / 8.4 / 14    277 / 282 / 288 -> 11 / 20 / 39      609 / 621 / 635 -> 40 / 65 / 116
//   Q4_KH   322 / 335 / 14 -> 6.5 / 7.6 / 11     445 / 446 / 22 ->  10 / 17 / 21      827 / 855 / 994 -> 32 / 52 /  -
//   f16     265 / 266 / 10 -> 7.1 / 7.6 /  -     271 / 271 / 16 ->  12 / 13 /  -      610 / 611 / 610 -> 38 / 43 /  -
// Weights that are known to be resident are requested before the predecessor has ended: 1.0 to 1.4 us less (Q8_0H, N = 3072: 3.9 / 5.1 / 7.8).
// Q8_0F at 2048 rows, N = K = 3072: 1416 -> 468.  What is left to the bytes of W (Q8_0H, 9216 x 3072: 4.6 us) is a CTA's start, its first
// loads and the sum over its warps.
#include "dequant.cuh"
#include "common.cuh"

namespace {

using namespace rcu_dequant;

enum { RW_F16 = 0, RW_Q8H = 1, RW_Q8F = 2, RW_Q4K = 3 };

struct RowsWeights {
    const unsigned char* codes;   // f16 values, int8 codes or nibble bytes
    const void* scales;           // Q8: block scales; Q4_KH: 12-byte (scale, min) packs
    const __half* d;              // Q4_KH super-block scale and min
    const __half* dmin;
};

constexpr int kRowsWarps = 8;

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// What a lane holds of one weight row of a chunk, as loaded: runs of eight elements, each with the eight elements of a token row that it
// meets.  CHUNK elements of a row are shared by the four lanes of a quad.  A lane takes sixteen consecutive elements, not more: the
// quad's loads of a token row then lie in one line of L1 (with 32 or 64 consecutive elements per lane they touch two or four, and at
// sixteen token rows those look-ups cost more than the weights).
//   f16     64 wide, lane t: elements 16 t .. 16 t + 15
//   Q8_0H  128 wide, lane t: elements 16 t .. of both halves
//   Q8_0F   64 wide, lane t: elements 8 t .. 8 t + 7 of both blocks, so that a product stays inside one block
//   Q4_KH  128 wide (half a super-block), lane t: sixteen bytes of the 32 whose nibbles are sub-blocks 2 (t / 2) and 2 (t / 2) + 1
template <int WT> struct RowRaw;
template <> struct RowRaw<RW_F16> {
    static constexpr int CHUNK = 64, RUNS = 2;
    uint4 v[2];
};
template <> struct RowRaw<RW_Q8H> {
    static constexpr int CHUNK = 128, RUNS = 4;
    uint4 v[2];
    __half d[2];
};
template <> struct RowRaw<RW_Q8F> {
    static constexpr int CHUNK = 64, RUNS = 2;
    uint2 v[2];
    float d[2];
};
template <> struct RowRaw<RW_Q4K> {
    static constexpr int CHUNK = 128, RUNS = 4;
    uint4 v;
    uint32_t pack[3];
    __half d, dmin;
};

// first element of run u
template <int WT> __device__ __forceinline__ int run_at(int c, int t, int u) {
    if constexpr (WT == RW_F16) return c * 64 + 16 * t + 8 * u;
    else if constexpr (WT == RW_Q8H) return c * 128 + 64 * (u >> 1) + 16 * t + 8 * (u & 1);
    else if constexpr (WT == RW_Q8F) return c * 64 + 32 * u + 8 * t;
    else return c * 128 + 64 * (t >> 1) + 32 * (u >> 1) + 16 * (t & 1) + 8 * (u & 1);
}

template <int WT> __device__ __forceinline__ RowRaw<WT> load_row(const RowsWeights& w, size_t row, int c, int t, int K) {
    RowRaw<WT> r;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    if constexpr (WT == RW_Q4K) {          // K is a multiple of 256: every chunk is whole
        const size_t sb = row * (size_t)(K >> 8) + (c >> 1);
        r.v = ld_stream_v4(w.codes + sb * 128 + (c & 1) * 64 + 16 * t);
        const uint32_t* p = reinterpret_cast<const uint32_t*>(w.scales) + sb * 3;
        r.pack[0] = __ldg(p);
        r.pack[1] = __ldg(p + 1);
        r.pack[2] = __ldg(p + 2);
        r.d = w.d[sb];
        r.dmin = w.dmin[sb];
    } else if constexpr (WT == RW_Q8H) {   // K is a multiple of 32: a block is whole or absent
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int k = run_at<WT>(c, t, 2 * j);
            const bool in = k < K;
            r.v[j] = in ? ld_stream_v4(w.codes + row * (size_t)K + k) : zero;
            r.d[j] = in ? reinterpret_cast<const __half*>(w.scales)[row * (size_t)(K >> 5) + (k >> 5)] : __float2half_rn(0.f);
        }
    } else {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int k = run_at<WT>(c, t, u);
            const bool in = k < K;         // K is a multiple of 32 (Q8_0F) or 8 (f16): a run is whole or absent
            if constexpr (WT == RW_F16) {
                r.v[u] = in ? ld_stream_v4(w.codes + (row * (size_t)K + k) * 2) : zero;
            } else {
                r.v[u] = in ? *reinterpret_cast<const uint2*>(w.codes + row * (size_t)K + k) : make_uint2(0u, 0u);
                r.d[u] = in ? reinterpret_cast<const float*>(w.scales)[row * (size_t)(K >> 5) + (k >> 5)] : 0.f;
            }
        }
    }
    return r;
}

// the eight f16 values of run u
template <int WT> __device__ __forceinline__ uint4 unpack_run(const RowRaw<WT>& r, int u, int c, int t) {
    if constexpr (WT == RW_F16) {
        return r.v[u];
    } else if constexpr (WT == RW_Q8H) {
        const uint4 q = r.v[u >> 1];
        const __half2 d = __half2half2(r.d[u >> 1]);
        return u & 1 ? dequant8_q8(q.z, q.w, d) : dequant8_q8(q.x, q.y, d);
    } else if constexpr (WT == RW_Q8F) {       // the codes themselves
        return dequant8_q8(r.v[u].x, r.v[u].y, __float2half2_rn(1.0f));
    } else {
        const int j = 2 * (t >> 1) + (u >> 1);         // sub-block of the half
        uint32_t sc, mn;
        if ((c & 1) == 0) {                            // ops/matmul/quantized.rs:158-204
            sc = (r.pack[0] >> (8 * j)) & 63u;
            mn = (r.pack[1] >> (8 * j)) & 63u;
        } else {
            const uint32_t low = r.pack[2] >> (8 * j);
            sc = (low & 0xFu) | ((r.pack[0] >> (8 * j + 6) & 3u) << 4);
            mn = (low >> 4 & 0xFu) | ((r.pack[1] >> (8 * j + 6) & 3u) << 4);
        }
        const __half2 mul = __half2half2(__hmul_rn(__uint2half_rn(sc), r.d)), neg = __half2half2(__hneg(__hmul_rn(__uint2half_rn(mn), r.dmin)));
        const uint32_t x0 = u & 1 ? r.v.z : r.v.x, x1 = u & 1 ? r.v.w : r.v.y;
        return u >= 2 ? dequant8_q4(x0 >> 4, x1 >> 4, mul, neg) : dequant8_q4(x0, x1, mul, neg);
    }
}

// NT: tiles of eight token rows, RT: tiles of sixteen weight rows, PF: chunks of weights a warp has requested ahead
template <int WT, int NT, int RT, int PF>
__global__ void __launch_bounds__(kRowsWarps * 32)
gemm_rows_kernel(const RowsWeights w, const __half* __restrict__ x, const __half* __restrict__ bias, __half* __restrict__ out, int M, int N, int K, int early) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!early) asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float red[kRowsWarps][16][NT * 8 + 1];      // one row tile at a time
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * RT * 16, m0 = blockIdx.y * NT * 8;
    const int chunks = (K + RowRaw<WT>::CHUNK - 1) / RowRaw<WT>::CHUNK;
    size_t rows[RT][2];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h) rows[r][h] = (size_t)min(n0 + r * 16 + h * 8 + g, N - 1);       // rows beyond N: computed, not stored
    RowRaw<WT> raw[PF][RT][2];
    auto fetch = [&](int slot, int c) {
        if (c >= chunks) return;
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int h = 0; h < 2; ++h) raw[slot][r][h] = load_row<WT>(w, rows[r][h], c, t, K);
    };
#pragma unroll
    for (int p = 0; p < PF; ++p) fetch(p, warp + p * kRowsWarps);
    // early: the weights stay as they are (the resolver knows; a caller's rcu_set_constant_weights speaks of matrix-vector products only); x may
    // be the predecessor's output
    if (early) asm volatile("griddepcontrol.wait;" ::: "memory");

    float acc[RT][NT][4];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[r][n][e] = 0.f;

    for (int c0 = warp; c0 < chunks; c0 += PF * kRowsWarps) {
#pragma unroll
        for (int p = 0; p < PF; ++p) {
            const int c = c0 + p * kRowsWarps;
            if (c >= chunks) break;
#pragma unroll
            for (int u = 0; u < RowRaw<WT>::RUNS; ++u) {
                uint4 wv[RT][2];
#pragma unroll
                for (int r = 0; r < RT; ++r)
#pragma unroll
                    for (int h = 0; h < 2; ++h) wv[r][h] = unpack_run<WT>(raw[p][r][h], u, c, t);
                const int k = run_at<WT>(c, t, u);
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const int tok = m0 + n * 8 + g;
                    uint4 xv = make_uint4(0u, 0u, 0u, 0u);
                    if (tok < M && k < K) xv = *reinterpret_cast<const uint4*>(x + (size_t)tok * K + k);
#pragma unroll
                    for (int r = 0; r < RT; ++r) {
                        const uint4 lo = wv[r][0], hi = wv[r][1];
                        if constexpr (WT == RW_Q8F) {
                            float part[4] = {0.f, 0.f, 0.f, 0.f};
                            mma_f16(part, lo.x, hi.x, lo.y, hi.y, xv.x, xv.y);
                            mma_f16(part, lo.z, hi.z, lo.w, hi.w, xv.z, xv.w);
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[r][n][e] = fmaf(raw[p][r][e >> 1].d[u], part[e], acc[r][n][e]);
                        } else {
                            mma_f16(acc[r][n], lo.x, hi.x, lo.y, hi.y, xv.x, xv.y);
                            mma_f16(acc[r][n], lo.z, hi.z, lo.w, hi.w, xv.z, xv.w);
                        }
                    }
                }
            }
            fetch(p, c + PF * kRowsWarps);
        }
    }
    // accumulator fragment: elements 0, 1 are row g and tokens 2 t, 2 t + 1, elements 2, 3 row g + 8
#pragma unroll
    for (int r = 0; r < RT; ++r) {
        if (r > 0) __syncthreads();
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) red[warp][(e >> 1) * 8 + g][n * 8 + 2 * t + (e & 1)] = acc[r][n][e];
        __syncthreads();
        for (int i = threadIdx.x; i < 16 * NT * 8; i += kRowsWarps * 32) {
            const int row = n0 + r * 16 + (i & 15), n = i >> 4;
            if (row >= N || m0 + n >= M) continue;
            float s = 0.f;
#pragma unroll
            for (int v = 0; v < kRowsWarps; ++v) s += red[v][i & 15][n];
            if (bias) s += __half2float(bias[row]);
            out[(size_t)(m0 + n) * N + row] = __float2half_rn(s);
        }
    }
}

template <int WT, int NT, int RT, int PF>
rcu_status launch_rows(rcu_device* dev, const RowsWeights& w, const void* x, const void* bias, void* y, int M, int N, int K) {
    constexpr int ROWS = RT * 16;
    const dim3 grid((N + ROWS - 1) / ROWS, (M + NT * 8 - 1) / (NT * 8));
    RCU_CUDA(dev, rcu_launch(dev, gemm_rows_kernel<WT, NT, RT, PF>, grid, kRowsWarps * 32, 0, w, (const __half*)x, (const __half*)bias, (__half*)y, M, N, K,
                             dev->resident_weights ? 1 : 0));
    RCU_LAUNCH_CHECK(dev);
    return RCU_OK;
}

template <int WT> rcu_status launch_rows_any(rcu_device* dev, const RowsWeights& w, const void* x, const void* bias, void* y, int M, int N, int K) {
    // two row tiles per warp halve the token loads; one puts a CTA on every SM when N is small
    const bool wide = N / 32 >= dev->sm_count * 3 / 2;
    if (M <= 8) return wide ? launch_rows<WT, 1, 2, 2>(dev, w, x, bias, y, M, N, K) : launch_rows<WT, 1, 1, 3>(dev, w, x, bias, y, M, N, K);
    if (M <= 16) return wide ? launch_rows<WT, 2, 2, 2>(dev, w, x, bias, y, M, N, K) : launch_rows<WT, 2, 1, 3>(dev, w, x, bias, y, M, N, K);
    if (M <= 32) return wide ? launch_rows<WT, 4, 2, 2>(dev, w, x, bias, y, M, N, K) : launch_rows<WT, 4, 1, 2>(dev, w, x, bias, y, M, N, K);
    if constexpr (WT == RW_Q8F) return launch_rows<WT, 8, 2, 1>(dev, w, x, bias, y, M, N, K);
    return RCU_ERR_UNSUPPORTED;
}

}  // namespace

// RCU_ERR_UNSUPPORTED: another kernel has to take the product
rcu_status rcu_gemm_rows_dispatch(rcu_device* dev, int lhs_dt, const void* w, int act_dt, const void* x, const void* bias, void* y, uint64_t M, uint64_t N,
                                  uint64_t K) {
    if (act_dt != RCU_F16 || M < 2 || N < 1 || K < 32) return RCU_ERR_UNSUPPORTED;
    if (M > 65535ull * 32 || N > 0x7fffffffull || K > 0x3fffffffull) return RCU_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) return RCU_ERR_UNSUPPORTED;
    DevGuard g(dev->ordinal);
    uint64_t off[4];
    rcu_dtype_segments(lhs_dt, N * K, off);
    const unsigned char* base = (const unsigned char*)w;
    RowsWeights rw{base, nullptr, nullptr, nullptr};
    const int m = (int)M, n = (int)N, k = (int)K;
    switch (lhs_dt) {
        case RCU_F16: return K % 8 ? RCU_ERR_UNSUPPORTED : launch_rows_any<RW_F16>(dev, rw, x, bias, y, m, n, k);
        case RCU_Q8_0H:
        case RCU_Q8_0F:
            if (K % 32) return RCU_ERR_UNSUPPORTED;
            rw.scales = base + off[1];
            return lhs_dt == RCU_Q8_0H ? launch_rows_any<RW_Q8H>(dev, rw, x, bias, y, m, n, k) : launch_rows_any<RW_Q8F>(dev, rw, x, bias, y, m, n, k);
        case RCU_Q4_KH:
            if (K % 256) return RCU_ERR_UNSUPPORTED;
            rw.scales = base + off[1];
            rw.dmin = (const __half*)(base + off[2]);
            rw.d = (const __half*)(base + off[3]);
            return launch_rows_any<RW_Q4K>(dev, rw, x, bias, y, m, n, k);
        default: return RCU_ERR_UNSUPPORTED;
    }
}
