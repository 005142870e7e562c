// Chains of small ops around the products of an f16 model that compute in f32 between two casts, each as one kernel.
#pragma once
#include "attention.cuh"

#ifdef __CUDACC__
// gelu or silu between two casts
__device__ __forceinline__ float chain_act(int act, float x) {
    if (act == RCU_GELU) return (0.5f * x) * (1.0f + tanhf((0.7978846f * x) * (1.0f + (0.044715f * x) * x)));      // the f32 form of unary gelu
    return x / (1.0f + expf(-x));
}
#endif

// out = f16(norm(f32(x)))  (nn's LayerNorm / RMSNorm: cast, norm, cast); scale and bias f32
rcu_status rcu_norm_half(rcu_device* dev, int kind, const void* x, const void* scale, const void* bias, float eps, void* out, uint64_t rows, uint64_t N);
// out = f16(act(f32(x)))
rcu_status rcu_act_half(rcu_device* dev, int act, const void* x, void* out, uint64_t n);
// out[t, c] = act(x[c, t]) + add[t, c], x [C, T] and add [T, C] f32, out f32 or (half) rounded to f16: what a convolution's output goes through on its way to
// rows of tokens
rcu_status rcu_act_rows(rcu_device* dev, int act, const float* x, const float* add, void* out, bool half, uint64_t T, uint64_t C);
// out = up * f16(act(f32(gate))) of rows that hold gate, then up
rcu_status rcu_glu_half(rcu_device* dev, int act, const void* x, void* out, uint64_t rows, uint64_t F);
// Heads out of rows: out[h, t, :] = src[t, h, :], rotated as rcu_rope does between casts to f32 and back (rope_dim 0: as they are)
struct HeadsRope {
    uint32_t dim = 0;
    float base = 0.f;
    uint32_t offset = 0;
    const void* table = nullptr;        // of rcu_heads_angles for these tokens
};
// [tokens][dim / 2] cos, sin as floats
rcu_status rcu_heads_angles(rcu_device* dev, const HeadsRope& rope, uint32_t tokens, void* table);
rcu_status rcu_heads_half(rcu_device* dev, const HeadRows& src, const HeadRows& dst, uint32_t heads, uint32_t tokens, uint32_t D, const HeadsRope& rope);

// A Linear with what follows it in the graph, on the tensor cores (gemm_tc.cu, gemm_tc2.cu): f16, out = f16(x W^T + bias), then gelu or silu between
// casts, or the addition to a residual; or (f16 and bf16) out = up * act(gate) of a product whose columns are gate, then up.
struct LinearChain {
    const void* bias = nullptr;         // in the activations' type
    const float* bias32 = nullptr;      // in f32, to be rounded to it
    const void* resid = nullptr;
    int op = -1, glu = -1;              // RCU_GELU, RCU_SILU
    uint64_t x_pitch = 0;               // of the activations' rows, 0: K
};
bool rcu_gemm_tc_chain_takes(rcu_device* dev, int w_dt, uint64_t M, uint64_t N, uint64_t K, bool glu, bool act);
rcu_status rcu_gemm_tc_chain(rcu_device* dev, int w_dt, const void* w, const void* x, void* y, uint64_t M, uint64_t N, uint64_t K, const LinearChain& c);

// The addition to a residual behind an f32 Linear that gemm_parts_f32.cu runs, where that pays: y = (x W^T + bias) + resid, each rounded as the ops by themselves do
bool rcu_gemm_parts_f32_takes(rcu_device* dev, uint64_t M, uint64_t N, uint64_t K);
rcu_status rcu_gemm_parts_f32_resid(rcu_device* dev, const void* w, const void* x, const void* bias, const void* resid, void* y, uint64_t M, uint64_t N, uint64_t K);

// Linears of the same sizes over the same rows, in one launch: the projections of an attention, each too small to fill the device.  q, k and v; a fourth
// Linear over the same rows runs by itself (every member's tensor map is 128 bytes of each launch's arguments).
constexpr int kGroupLinears = 3;
struct LinearGroup {
    int n = 0;
    uint64_t M = 0, N = 0, K = 0;
    const void* x = nullptr;
    const void* w[kGroupLinears] = {};          // in the activations' type
    const void* bias[kGroupLinears] = {};       // likewise, nullable
    const float* bias32[kGroupLinears] = {};    // f16 activations: in f32, to be rounded first, nullable
    void* out[kGroupLinears] = {};
};
// RCU_ERR_UNSUPPORTED: nothing was launched; sizes or alignments that the kernel does not take, or products that fill the device one by one
rcu_status rcu_gemm_tc_group(rcu_device* dev, const LinearGroup& g);            // f16
rcu_status rcu_gemm_parts_f32_group(rcu_device* dev, const LinearGroup& g);     // f32

// The Linears of a resolve whose weights are converted once per product (gemm_tc.cu, matmul.cu), converted together: small matrices, in one launch
struct DequantItem {
    const void* src;                    // Q8_0 segments
    void* dst;
    uint64_t numel;
};
constexpr int kDequantItems = 32;       // of one launch
rcu_status rcu_dequantize_items(rcu_device* dev, int dt, const DequantItem* items, int n);
// The conversion that dev->next_conversion describes, launched beside the kernel before it, which must be one that triggers its dependents behind
// its own wait and neither writes these weights nor uses the destination.  RCU_ERR_UNSUPPORTED: nothing was launched.
rcu_status rcu_dequantize_beside(rcu_device* dev, const rcu_device::NextConversion& c);
// whether a Linear over M rows of activations converts its weights of this type in a launch of its own
bool rcu_linear_converts(int w_dt, int act_dt, uint64_t M, uint64_t N, uint64_t K);
// ... of Q8_0H weights under f16 activations, and the product over them is the pair kernel's
bool rcu_linear_converts_beside(rcu_device* dev, uint64_t M, uint64_t N, uint64_t K);
