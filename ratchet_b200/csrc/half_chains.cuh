// Chains of small ops around the products of an f16 model that compute in f32 between two casts, each as one kernel.
#pragma once
#include "attention.cuh"

// out = f16(norm(f32(x)))  (nn's LayerNorm / RMSNorm: cast, norm, cast); scale and bias f32
rcu_status rcu_norm_half(rcu_device* dev, int kind, const void* x, const void* scale, const void* bias, float eps, void* out, uint64_t rows, uint64_t N);
// out = f16(act(f32(x)))
rcu_status rcu_act_half(rcu_device* dev, int act, const void* x, void* out, uint64_t n);
// out = up * f16(act(f32(gate))) of rows that hold gate, then up
rcu_status rcu_glu_half(rcu_device* dev, int act, const void* x, void* out, uint64_t rows, uint64_t F);
// Heads out of rows: out[h, t, :] = src[t, h, :], rotated as rcu_rope does between casts to f32 and back (rope_dim 0: as they are)
struct HeadsRope {
    uint32_t dim = 0;
    float base = 0.f;
    uint32_t offset = 0;
};
rcu_status rcu_heads_half(rcu_device* dev, const HeadRows& src, const HeadRows& dst, uint32_t heads, uint32_t tokens, uint32_t D, const HeadsRope& rope);
