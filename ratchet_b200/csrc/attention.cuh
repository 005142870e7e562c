// Softmax attention of a block over f16 queries, keys and values that lie in memory as their producers left them: element (position, head,
// feature) at position * row + head * head_pitch + feature.
#pragma once
#include "common.cuh"

struct HeadRows {
    const void* data = nullptr;     // first element
    uint64_t head = 0, row = 0;     // pitches in elements
};

struct AttentionArgs {
    HeadRows q, k, v;
    void* out;                      // [T, H, E] f16
    int H, T, L, D, E;
    const float* scale32[1];        // factor of the scores in f32, nullable
    const __half* scale16[2];       // factors that queries and keys carry in f16, nullable
    const __half* mask;             // added to the scores in f16, [T, L], nullable
};

// RCU_ERR_UNSUPPORTED: sizes or alignments the kernel does not take (nothing has been launched)
rcu_status rcu_attention_f16(rcu_device* dev, const AttentionArgs& a);
bool rcu_attention_f16_takes(const rcu_device* dev, const AttentionArgs& a);

// The same in f32, the factors of queries and keys as f32 tensors of one element
struct Attention32Args {
    HeadRows q, k, v;
    void* out;                      // [T, H, E] f32
    int H, T, L, D, E;
    const float* scale[2];          // nullable
};
rcu_status rcu_attention_f32(rcu_device* dev, const Attention32Args& a);
bool rcu_attention_f32_takes(const rcu_device* dev, const Attention32Args& a);
