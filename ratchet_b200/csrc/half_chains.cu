// One kernel each for the chains cast -> op in f32 -> cast that an f16 graph holds around its products (ratchet-nn/src/norm.rs:37-69,
// rope.rs:24-45, phi3/attn.rs:95-117, phi3/mlp.rs:31-39, whisper/mlp.rs:18-22).  The resolver (graph_fusion.cuh) sends them here; the
// arithmetic is that of the ops' own f32 kernels, so results are the unfused chain's.
//
// All are bound by memory, or by their launch: a chain of three kernels read and wrote its f32 intermediates, six times the bytes of
// the f16 rows.  Measured on B200 at 1000 rows of 3072 (us per chain, unfused -> one kernel): norm 14 -> 4, rotation of 32 heads with
// its slice and permutes 25 -> 5, silu gate of 2 x 8192 features 58 -> 12.
#include <cmath>

#include "half_chains.cuh"

namespace {

struct alignas(16) Half8 { __half v[8]; };

// CTA = one row of up to 256 * 8 * PER features, kept in registers
template <int PER>
__global__ void __launch_bounds__(256)
norm_half_kernel(const __half* __restrict__ x, const float* __restrict__ scale, const float* __restrict__ bias, __half* __restrict__ out, int N, float eps, int layer) {
    rcu_kernel_entry();
    __shared__ float scratch[2][8];
    const __half* xr = x + (size_t)blockIdx.x * N;
    float v[PER][8];
    float s = 0.f, s2 = 0.f;
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int j = (threadIdx.x + p * 256) * 8;
        if (j >= N) continue;
        const Half8 h = *reinterpret_cast<const Half8*>(xr + j);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[p][e] = __half2float(h.v[e]);
            s += v[p][e];
            s2 += v[p][e] * v[p][e];
        }
    }
    s = warp_sum(s);
    s2 = warp_sum(s2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        scratch[0][warp] = s;
        scratch[1][warp] = s2;
    }
    __syncthreads();
    s = warp_sum(lane < 8 ? scratch[0][lane] : 0.f);
    s2 = warp_sum(lane < 8 ? scratch[1][lane] : 0.f);
    const float n = (float)N, mu = layer ? s / n : 0.f;
    const float var = layer ? s2 / n - mu * mu : s2 / n;
    const float rstd = 1.0f / sqrtf(var + eps);
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int j = (threadIdx.x + p * 256) * 8;
        if (j >= N) continue;
        Half8 o;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float4 g = *reinterpret_cast<const float4*>(scale + j + 4 * q);
            const float4 b = bias ? *reinterpret_cast<const float4*>(bias + j + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float gv[4] = {g.x, g.y, g.z, g.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) o.v[4 * q + e] = __float2half_rn(__fadd_rn(__fmul_rn(__fmul_rn(v[p][4 * q + e] - mu, rstd), gv[e]), bv[e]));
        }
        *reinterpret_cast<Half8*>(out + (size_t)blockIdx.x * N + j) = o;
    }
}

__global__ void __launch_bounds__(256) act_half_kernel(const __half* __restrict__ x, __half* __restrict__ out, size_t n8, int act) {
    rcu_kernel_entry();
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n8; i += (size_t)gridDim.x * 256) {
        const Half8 h = reinterpret_cast<const Half8*>(x)[i];
        Half8 o;
#pragma unroll
        for (int e = 0; e < 8; ++e) o.v[e] = __float2half_rn(chain_act(act, __half2float(h.v[e])));
        reinterpret_cast<Half8*>(out)[i] = o;
    }
}

// 32 x 32 pieces turned around in shared memory.  Launch-bound: whisper/encoder.rs:49-55 has unary, permute, addition and cast here, 5 us each
// (Whisper-tiny's encoder: f16 244 us with them apart, 240 in one; f32 548, 540).
template <class Out>
__global__ void __launch_bounds__(256) act_rows_kernel(const float* __restrict__ x, const float* __restrict__ add, Out* __restrict__ out, int T, int C, int act) {
    rcu_kernel_entry();
    __shared__ float turn[32][33];
    const int t0 = blockIdx.x * 32, c0 = blockIdx.y * 32, i = threadIdx.x & 31, j = threadIdx.x >> 5;
    float v[4], p[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        const int c = c0 + j + 8 * n, t = t0 + j + 8 * n;
        v[n] = c < C && t0 + i < T ? x[(size_t)c * T + t0 + i] : 0.f;
        p[n] = t < T && c0 + i < C ? add[(size_t)t * C + c0 + i] : 0.f;
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) turn[j + 8 * n][i] = chain_act(act, v[n]);
    __syncthreads();
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        const int t = t0 + j + 8 * n;
        if (t < T && c0 + i < C) out[(size_t)t * C + c0 + i] = from_f32<Out>(turn[i][j + 8 * n] + p[n]);
    }
}

__global__ void __launch_bounds__(256) glu_half_kernel(const __half* __restrict__ x, __half* __restrict__ out, size_t n8, int f8, int act) {
    rcu_kernel_entry();
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n8; i += (size_t)gridDim.x * 256) {
        const size_t row = i / f8, j = i - row * f8;
        const Half8 g = reinterpret_cast<const Half8*>(x)[row * 2 * f8 + j], u = reinterpret_cast<const Half8*>(x)[row * 2 * f8 + f8 + j];
        Half8 o;
#pragma unroll
        for (int e = 0; e < 8; ++e) o.v[e] = __hmul_rn(u.v[e], __float2half_rn(chain_act(act, __half2float(g.v[e]))));
        reinterpret_cast<Half8*>(out)[i] = o;
    }
}

// Thread = one rotation pair of one position (as rcu_rope, cpu/rope.rs:38-41).  Some 200 double-precision operations, so that a prompt of 1000
// tokens takes 3 us; inside the rotation of every layer's queries and keys they were most of its 13 us (5.3 without).
__global__ void __launch_bounds__(128) heads_angles_kernel(float2* __restrict__ table, int n, int half, float ln_base, int offset) {
    rcu_kernel_entry();
    const int idx = blockIdx.x * 128 + threadIdx.x;
    if (idx >= n) return;
    const int s = idx / half, i = idx - s * half;
    const float ex = -(float)i * ln_base / (float)half;
    const float inv = (float)exp((double)ex), th = (float)(s + offset) * inv;
    double sd, cd;
    sincos((double)th, &sd, &cd);
    table[idx] = make_float2((float)cd, (float)sd);
}

// Thread = eight consecutive rotation pairs of one position: their angles once, then every head this thread visits
__global__ void __launch_bounds__(128)
heads_rope_kernel(const __half* __restrict__ x, __half* __restrict__ out, size_t xh, size_t xr, size_t oh, size_t orow, int H, int T, int D, int dim, const float2* __restrict__ table) {
    rcu_kernel_entry();
    const int half = dim >> 1, hv = half / 8, idx = blockIdx.x * 128 + threadIdx.x;
    if (idx < T * hv) {
        const int s = idx / hv, i0 = (idx - s * hv) * 8;
        float sn[8], cs[8];
        const float4* row = reinterpret_cast<const float4*>(table + (size_t)s * half + i0);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float4 v = row[e];
            cs[2 * e] = v.x;
            sn[2 * e] = v.y;
            cs[2 * e + 1] = v.z;
            sn[2 * e + 1] = v.w;
        }
#pragma unroll 2
        for (int h = blockIdx.y; h < H; h += gridDim.y) {
            const __half* p = x + h * xh + s * xr + i0;
            __half* q = out + h * oh + s * orow + i0;
            const Half8 a = *reinterpret_cast<const Half8*>(p), b = *reinterpret_cast<const Half8*>(p + half);
            Half8 ra, rb;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float x1 = __half2float(a.v[e]), x2 = __half2float(b.v[e]);
                ra.v[e] = __float2half_rn(__fsub_rn(__fmul_rn(x1, cs[e]), __fmul_rn(x2, sn[e])));
                rb.v[e] = __float2half_rn(__fadd_rn(__fmul_rn(x1, sn[e]), __fmul_rn(x2, cs[e])));
            }
            *reinterpret_cast<Half8*>(q) = ra;
            *reinterpret_cast<Half8*>(q + half) = rb;
        }
    }
    const int tv = (D - dim) / 8;                // features that are not rotated
    if (idx < T * tv) {
        const int s = idx / tv, i = dim + (idx - s * tv) * 8;
        for (int h = blockIdx.y; h < H; h += gridDim.y)
            *reinterpret_cast<Half8*>(out + h * oh + s * orow + i) = *reinterpret_cast<const Half8*>(x + h * xh + s * xr + i);
    }
}

__global__ void __launch_bounds__(256)
heads_copy_kernel(const __half* __restrict__ x, __half* __restrict__ out, size_t xh, size_t xr, size_t oh, size_t orow, int H, int T, int d8) {
    rcu_kernel_entry();
    const size_t n = (size_t)H * T * d8;
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
        const size_t r = i / d8, h = r / T, t = r - h * T, d = (i - r * d8) * 8;
        *reinterpret_cast<Half8*>(out + h * oh + t * orow + d) = *reinterpret_cast<const Half8*>(x + h * xh + t * xr + d);
    }
}

bool aligned16(std::initializer_list<const void*> ps) {
    uintptr_t u = 0;
    for (const void* p : ps) u |= reinterpret_cast<uintptr_t>(p);
    return (u & 15) == 0;
}

}  // namespace

rcu_status rcu_norm_half(rcu_device* dev, int kind, const void* x, const void* scale, const void* bias, float eps, void* out, uint64_t rows, uint64_t N) {
    if (N % 8 || N > 8192 || rows > 0x7fffffffull || rows == 0 || !aligned16({x, scale, bias, out})) return RCU_ERR_UNSUPPORTED;
    const int layer = kind == RCU_LAYER_NORM;
#define RCU_NH(PER) rcu_launch(dev, norm_half_kernel<PER>, (unsigned)rows, 256, 0, (const __half*)x, (const float*)scale, (const float*)bias, (__half*)out, (int)N, eps, layer)
    RCU_CUDA(dev, N <= 2048 ? RCU_NH(1) : N <= 4096 ? RCU_NH(2) : RCU_NH(4));
#undef RCU_NH
    RCU_LAUNCH_CHECK(dev);
    return RCU_OK;
}

rcu_status rcu_act_rows(rcu_device* dev, int act, const float* x, const float* add, void* out, bool half, uint64_t T, uint64_t C) {
    if (T > 0x7fffffffull || (C + 31) / 32 > 65535) return RCU_ERR_UNSUPPORTED;
    const dim3 grid((unsigned)((T + 31) / 32), (unsigned)((C + 31) / 32));
    if (half) RCU_CUDA(dev, rcu_launch(dev, act_rows_kernel<__half>, grid, 256, 0, x, add, (__half*)out, (int)T, (int)C, act));
    else RCU_CUDA(dev, rcu_launch(dev, act_rows_kernel<float>, grid, 256, 0, x, add, (float*)out, (int)T, (int)C, act));
    RCU_LAUNCH_CHECK(dev);
    return RCU_OK;
}

rcu_status rcu_act_half(rcu_device* dev, int act, const void* x, void* out, uint64_t n) {
    if (n % 8 || n == 0 || !aligned16({x, out})) return RCU_ERR_UNSUPPORTED;
    RCU_CUDA(dev, rcu_launch(dev, act_half_kernel, (unsigned)grid_for(n / 8, 256, dev->sm_count * 16), 256, 0, (const __half*)x, (__half*)out, (size_t)(n / 8), act));
    RCU_LAUNCH_CHECK(dev);
    return RCU_OK;
}

rcu_status rcu_glu_half(rcu_device* dev, int act, const void* x, void* out, uint64_t rows, uint64_t F) {
    if (F % 8 || F == 0 || rows == 0 || F > 0x7fffffffull || !aligned16({x, out})) return RCU_ERR_UNSUPPORTED;
    const size_t n8 = rows * (F / 8);
    RCU_CUDA(dev, rcu_launch(dev, glu_half_kernel, (unsigned)grid_for(n8, 256, dev->sm_count * 16), 256, 0, (const __half*)x, (__half*)out, n8, (int)(F / 8), act));
    RCU_LAUNCH_CHECK(dev);
    return RCU_OK;
}

rcu_status rcu_heads_angles(rcu_device* dev, const HeadsRope& rope, uint32_t tokens, void* table) {
    const uint64_t n = (uint64_t)tokens * (rope.dim / 2);
    if (rope.dim % 16 || n == 0 || n > 0x7fffffffull) return RCU_ERR_UNSUPPORTED;
    RCU_CUDA(dev, rcu_launch(dev, heads_angles_kernel, (unsigned)((n + 127) / 128), 128, 0, (float2*)table, (int)n, (int)(rope.dim / 2), logf(rope.base), (int)rope.offset));
    RCU_LAUNCH_CHECK(dev);
    return RCU_OK;
}

rcu_status rcu_heads_half(rcu_device* dev, const HeadRows& src, const HeadRows& dst, uint32_t H, uint32_t T, uint32_t D, const HeadsRope& rope) {
    if (D % 8 || D == 0 || H == 0 || T == 0 || (src.head | src.row | dst.head | dst.row) % 8 || !aligned16({src.data, dst.data}) || (uint64_t)T * D > 0x7fffffffull)
        return RCU_ERR_UNSUPPORTED;
    const __half* x = (const __half*)src.data;
    __half* o = (__half*)const_cast<void*>(dst.data);
    if (rope.dim == 0) {
        RCU_CUDA(dev, rcu_launch(dev, heads_copy_kernel, (unsigned)grid_for((uint64_t)H * T * (D / 8), 256, dev->sm_count * 16), 256, 0, x, o, (size_t)src.head, (size_t)src.row,
                                 (size_t)dst.head, (size_t)dst.row, (int)H, (int)T, (int)(D / 8)));
    } else {
        if (rope.dim % 16 || rope.dim > D || !rope.table) return RCU_ERR_UNSUPPORTED;
        const int per_row = std::max<int>(rope.dim / 16, (D - rope.dim) / 8), gx = ((int)T * per_row + 127) / 128;
        const int want = (dev->sm_count * 16 + gx - 1) / gx;
        RCU_CUDA(dev, rcu_launch(dev, heads_rope_kernel, dim3(gx, (unsigned)std::max(1, std::min<int>((int)H, want))), 128, 0, x, o, (size_t)src.head, (size_t)src.row,
                                 (size_t)dst.head, (size_t)dst.row, (int)H, (int)T, (int)D, (int)rope.dim, (const float2*)rope.table));
    }
    RCU_LAUNCH_CHECK(dev);
    return RCU_OK;
}
