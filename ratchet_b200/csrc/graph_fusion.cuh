// Subgraphs of a prompt that the resolver runs as one kernel (included by graph.cu).
//
// Only nodes that nothing outside the graph holds, and that a single op consumes, are passed over: they get no buffer and no kernel.
// What is recognised (T > 1 positions; single tokens keep one kernel per op):
//   attention    permute(softmax(f32(scores [+ mask])) v), scores = f16(scale * f32(q) f32(k)^T) with keys and values that a cache returns or
//                that are given (phi3/attn.rs:119-157), or (dk q)(dk k^T) in f16 (whisper/mha.rs:92-127); permutes of views of
//                q, k and v become strides, and a cache that only feeds the attention is appended to but not copied out
//   attention32  permute(softmax((dk q)(dk k)^T) v) in f32 (the same with f32 activations, whose casts are no nodes)
//   heads        cast(rope(cast(permute(view(slice))))), and permute(view(slice)) in front of a cache: straight into the cache's rows
//   linear       a product with its bias's cast, gelu or silu between casts or the addition to the residual behind it; the product of a glu
//                (bf16's too); the addition to the residual behind an f32 product as well
//   rows         [cast](permute(gelu or silu(x)) + positions) in f32, a convolution's [1, C, T] on its way to rows of tokens (whisper/encoder.rs:108-122)
//   norm         cast(norm(cast x));   act: cast(gelu or silu(cast x));   glu: up * cast(silu(cast gate)) of the halves of one tensor
// A subgraph whose sizes or alignment a kernel does not take stays as it is.
#pragma once

namespace fusion {

enum Kind { NONE = 0, ATTENTION, ATTENTION32, HEADS, APPEND, NORM, ACT, GLU, LINEAR, ROWS };

// element (position t, head h, feature d) of a [1, heads, T, D] operand at base[offset + h * head + t * row + d]
struct Heads {
    rcu_lazy* base = nullptr;
    uint64_t offset = 0, head = 0, row = 0;
    HeadRows rows() const { return HeadRows{(const char*)base->storage->ptr + offset * 2, head, row}; }
};

struct Op {
    Kind kind = NONE;
    std::vector<rcu_lazy*> srcs;        // what the kernel reads
    Heads q, k, v;                      // HEADS and APPEND: q is the source
    rcu_lazy *mask = nullptr, *scale = nullptr, *scale_q = nullptr, *scale_k = nullptr;
    bool copied = false;                // APPEND: the source is an ordinary [1, H, T, D] tensor
    HeadsRope rope;
    uint32_t H = 0, T = 0, L = 0, D = 0, E = 0;
    rcu_lazy *w = nullptr, *x = nullptr, *bias = nullptr, *bias32 = nullptr, *resid = nullptr;      // LINEAR
    int act = -1, glu = -1;
    bool full = false;                  // f32 (with a residual)
    uint32_t x_col = 0;
    uint64_t M = 0, N = 0, K = 0;
};

// `t` exists only for its one consumer
inline bool inner(const rcu_lazy* t) { return !t->resolved() && t->refs.load() == 1; }
inline bool inner(const rcu_lazy* t, int kind, int32_t dt) { return inner(t) && t->kind == kind && t->dt == dt; }
inline bool permutes(const rcu_lazy* t, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return t->rank == 4 && t->u[0] == a && t->u[1] == b && t->u[2] == c && t->u[3] == d;
}

struct Pass {
    rcu_device* dev;
    const Order& order;
    static constexpr int kPlain = -1, kPassed = -2;
    std::deque<Op> ops;
    std::vector<int> role;                          // by position in the order: the op whose result the node is, or no kernel nor buffer (kPassed)
    struct Written { const rcu_lazy* t; const char *begin, *end; };      // begin null: not resolved
    std::vector<Written> written;                   // tensors that a node of this graph writes into, once per node

    int role_of(const rcu_lazy* t) const {
        const uint32_t at = order.at(t);
        return at == Order::kNone ? kPlain : role[at];
    }
    bool absorbed(const rcu_lazy* t) const { return role_of(t) == kPassed; }
    const Op* find(const rcu_lazy* t) const {
        const int r = role_of(t);
        return r < 0 ? nullptr : &ops[r];
    }
    // `root` becomes the op, the nodes behind it are passed over: unless one of them has a part already, or a node that comes between where
    // they stood and where the op runs may write into what the op reads (a cache's rows that the op's own appends write are not in `reads`)
    bool give(const rcu_lazy* root, Op&& op, const std::vector<rcu_lazy*>& seen, const std::vector<rcu_lazy*>& reads) {
        for (const rcu_lazy* t : seen)
            if (absorbed(t) || find(t)) return false;
        for (const rcu_lazy* t : reads)
            if (t && writes_to(t) > 0) return false;
        for (const rcu_lazy* t : seen) role[order.at(t)] = kPassed;
        role[order.at(root)] = (int)ops.size();
        ops.push_back(std::move(op));
        return true;
    }
    bool give(const rcu_lazy* root, Op&& op, const std::vector<rcu_lazy*>& seen) {
        const std::vector<rcu_lazy*> reads = op.srcs;
        return give(root, std::move(op), seen, reads);
    }

    // The operand [1, H, T, D] `x` as strides into the tensor behind its permute, view and slice, where these are its own; `seen` receives
    // the nodes passed over.  time_last: x is [1, H, D, T].
    static Heads strides(rcu_lazy* x, bool time_last, std::vector<rcu_lazy*>* seen, int32_t dt = RCU_F16) {
        const uint64_t H = x->shape[1], T = x->shape[time_last ? 3 : 2], D = x->shape[time_last ? 2 : 3];
        const bool perm = inner(x, K_PERMUTE, dt) && (time_last ? permutes(x, 0, 2, 3, 1) : permutes(x, 0, 2, 1, 3));
        if (!perm) {
            if (time_last) return Heads{};
            return Heads{x, 0, T * D, D};
        }
        rcu_lazy* y = x->srcs[0];                    // [1, T, H, D]
        seen->push_back(x);
        if (!inner(y, K_VIEW, dt)) return Heads{y, 0, D, H * D};
        rcu_lazy* z = y->srcs[0];
        seen->push_back(y);
        if (inner(z, K_SLICE, dt) && z->rank == 3 && z->shape[0] == 1 && z->shape[1] == T && z->shape[2] == H * D) {
            rcu_lazy* w = z->srcs[0];
            if (w->rank == 3 && w->shape[0] == 1 && w->shape[1] == T && z->a[0] == 0 && z->a[1] == 0) {
                seen->push_back(z);
                return Heads{w, z->a[2], D, w->shape[2]};
            }
        }
        return Heads{z, 0, D, H * D};
    }

    static bool vectors(const Heads& h) { return h.base && h.offset % 8 == 0 && h.head % 8 == 0 && h.row % 8 == 0 && aligned(h.base); }

    // the tensor whose memory `t` is
    static const rcu_lazy* viewed(const rcu_lazy* t) {
        while (!t->resolved() && t->kind == K_VIEW) t = t->srcs[0];
        return t;
    }

    // whether the kernels' 16-byte accesses fit: pool blocks do, a tensor over memory of the caller's may not
    static bool aligned(const rcu_lazy* t) {
        t = viewed(t);
        return !t->resolved() || (reinterpret_cast<uintptr_t>(t->storage->ptr) & 15) == 0;
    }

    // a cache that returns [1, H, L, D] and feeds only the attention: its tensor's rows in place
    Heads from_cache(rcu_lazy* x, std::vector<rcu_lazy*>* appends) const {
        if (!inner(x, K_CACHE, RCU_F16) || x->rank != 4 || x->u[0] != 2) return Heads{};
        const rcu_lazy* src = x->srcs[1];
        rcu_lazy* c = x->srcs[0];
        if (!c->resolved() || c->rank != 4 || c->shape[0] != 1 || !aligned(c) || writes_to(c) != 1) return Heads{};
        if (src->shape[0] != 1 || src->shape[1] != c->shape[1] || src->shape[3] != c->shape[3]) return Heads{};      // rcu_cache refuses it
        appends->push_back(x);
        return Heads{c, 0, c->shape[2] * c->shape[3], c->shape[3]};
    }

    // nodes of this graph that write into the memory of `t`
    int writes_to(const rcu_lazy* t) const {
        t = viewed(t);
        const char *begin = t->resolved() ? (const char*)t->storage->ptr : nullptr, *end = begin ? begin + t->nbytes() : nullptr;
        int n = 0;
        for (const Written& w : written) n += w.t == t || (begin && w.begin && begin < w.end && w.begin < end);
        return n;
    }

    bool attention(rcu_lazy* root) {
        if (root->dt != RCU_F16 || root->rank != 4 || !permutes(root, 0, 2, 1, 3) || root->shape[0] != 1) return false;
        std::vector<rcu_lazy*> seen, appends;
        rcu_lazy* pv = root->srcs[0];
        if (!inner(pv, K_MATMUL, RCU_F16) || pv->srcs.size() != 2 || pv->flags[0] || pv->flags[1] || pv->flags[2]) return false;
        rcu_lazy *w = pv->srcs[0], *v = pv->srcs[1];
        if (!inner(w, K_CAST, RCU_F16) || v->rank != 4 || w->rank != 4 || w->shape[0] != 1 || v->shape[0] != 1 || v->shape[1] != w->shape[1]) return false;
        rcu_lazy* sm = w->srcs[0];
        if (!inner(sm, K_SOFTMAX, RCU_F32) || sm->u[0] != 3) return false;
        rcu_lazy* full = sm->srcs[0];
        if (!inner(full, K_CAST, RCU_F32)) return false;
        seen.insert(seen.end(), {pv, w, sm, full});
        Op op;
        op.kind = ATTENTION;
        op.H = (uint32_t)w->shape[1];
        op.T = (uint32_t)w->shape[2];
        op.L = (uint32_t)w->shape[3];
        op.E = (uint32_t)v->shape[3];
        if (op.T < 2 || w->shape[2] > 0x7fffffffull || w->shape[3] > 0x7fffffffull) return false;
        rcu_lazy* z = full->srcs[0];
        if (inner(z, K_BINARY, RCU_F16) && z->op == RCU_ADD) {
            rcu_lazy *x = z->srcs[0], *m = z->srcs[1];
            const uint32_t r = m->rank;
            if (m->dt != RCU_F16 || r < 2 || m->shape[r - 2] != op.T || m->shape[r - 1] != op.L || m->numel() != (uint64_t)op.T * op.L) return false;
            op.mask = m;
            seen.push_back(z);
            z = x;
        }
        rcu_lazy *q, *k;
        bool k_cached = false;
        if (inner(z, K_CAST, RCU_F16)) {            // f16(scale * f32(q) f32(k)^T)
            rcu_lazy* mul = z->srcs[0];
            if (!inner(mul, K_BINARY, RCU_F32) || mul->op != RCU_MUL || mul->srcs[1]->numel() != 1 || mul->srcs[1]->dt != RCU_F32) return false;
            rcu_lazy* qk = mul->srcs[0];
            if (!inner(qk, K_MATMUL, RCU_F32) || qk->srcs.size() != 2 || qk->flags[0] || !qk->flags[1] || qk->flags[2]) return false;
            rcu_lazy *q32 = qk->srcs[0], *k32 = qk->srcs[1];
            if (!inner(q32, K_CAST, RCU_F32) || !inner(k32, K_CAST, RCU_F32)) return false;
            q = q32->srcs[0];
            k = k32->srcs[0];
            if (q->dt != RCU_F16 || k->dt != RCU_F16) return false;
            op.scale = mul->srcs[1];
            seen.insert(seen.end(), {z, mul, qk, q32, k32});
            if (q->rank != 4 || k->rank != 4 || q->shape[0] != 1 || q->shape[1] != op.H || q->shape[2] != op.T || k->shape[0] != 1 || k->shape[1] != op.H ||
                k->shape[2] != op.L || k->shape[3] != q->shape[3])
                return false;
            op.D = (uint32_t)q->shape[3];
            op.q = strides(q, false, &seen);
            op.k = from_cache(k, &appends);
            k_cached = op.k.base != nullptr;
            if (!k_cached) op.k = strides(k, false, &seen);
        } else if (inner(z, K_MATMUL, RCU_F16) && !op.mask && z->srcs.size() == 2 && !z->flags[0] && !z->flags[1] && !z->flags[2]) {     // (q dk)(k^T dk)
            rcu_lazy *qm = z->srcs[0], *km = z->srcs[1];
            for (rcu_lazy* t : {qm, km})
                if (!inner(t, K_BINARY, RCU_F16) || t->op != RCU_MUL || t->srcs[1]->numel() != 1 || t->srcs[1]->dt != RCU_F16 || t->rank != 4) return false;
            q = qm->srcs[0];
            k = km->srcs[0];
            op.scale_q = qm->srcs[1];
            op.scale_k = km->srcs[1];
            seen.insert(seen.end(), {z, qm, km});
            if (q->rank != 4 || k->rank != 4 || q->shape[0] != 1 || q->shape[1] != op.H || q->shape[2] != op.T || k->shape[0] != 1 || k->shape[1] != op.H ||
                k->shape[3] != op.L || k->shape[2] != q->shape[3])
                return false;
            op.D = (uint32_t)q->shape[3];
            op.q = strides(q, false, &seen);
            op.k = strides(k, true, &seen);
        } else {
            return false;
        }
        if (v->shape[2] != op.L) return false;
        op.v = from_cache(v, &appends);
        const bool v_cached = op.v.base != nullptr;
        if (!v_cached) op.v = strides(v, false, &seen);
        if (!vectors(op.q) || !vectors(op.k) || !vectors(op.v)) return false;
        AttentionArgs a{};
        a.q = HeadRows{nullptr, op.q.head, op.q.row};
        a.k = HeadRows{nullptr, op.k.head, op.k.row};
        a.v = HeadRows{nullptr, op.v.head, op.v.row};
        a.H = (int)op.H; a.T = (int)op.T; a.L = (int)op.L; a.D = (int)op.D; a.E = (int)op.E;
        a.mask = op.mask ? (const __half*)16 : nullptr;
        if (!rcu_attention_f16_takes(dev, a)) return false;
        std::vector<rcu_lazy*> reads = {op.q.base, op.mask, op.scale, op.scale_q, op.scale_k};
        if (!k_cached) reads.push_back(op.k.base);
        if (!v_cached) reads.push_back(op.v.base);
        op.srcs = {op.q.base, op.k.base, op.v.base};
        for (rcu_lazy* t : {op.mask, op.scale, op.scale_q, op.scale_k})
            if (t) op.srcs.push_back(t);
        op.srcs.insert(op.srcs.end(), appends.begin(), appends.end());       // these run before the attention and hold no buffer
        if (!give(root, std::move(op), seen, reads)) return false;
        for (rcu_lazy* t : appends) append(t);
        return true;
    }

    // the same in f32, without casts, mask or cache
    bool attention32(rcu_lazy* root) {
        if (root->dt != RCU_F32 || root->rank != 4 || !permutes(root, 0, 2, 1, 3) || root->shape[0] != 1) return false;
        std::vector<rcu_lazy*> seen;
        auto product = [&](rcu_lazy* t) { return inner(t, K_MATMUL, RCU_F32) && t->srcs.size() == 2 && !t->flags[0] && !t->flags[1] && !t->flags[2]; };
        rcu_lazy* pv = root->srcs[0];
        if (!product(pv)) return false;
        rcu_lazy *w = pv->srcs[0], *v = pv->srcs[1];
        if (!inner(w, K_SOFTMAX, RCU_F32) || w->u[0] != 3 || w->rank != 4 || w->shape[0] != 1) return false;
        rcu_lazy* z = w->srcs[0];
        if (!product(z)) return false;
        seen.insert(seen.end(), {pv, w, z});
        Op op;
        op.kind = ATTENTION32;
        const uint64_t H = w->shape[1], T = w->shape[2], L = w->shape[3];
        if (H > 65535 || T > 0x7fffffffull || L > 0x7fffffffull) return false;
        op.H = (uint32_t)H;
        op.T = (uint32_t)T;
        op.L = (uint32_t)L;
        rcu_lazy* side[2] = {z->srcs[0], z->srcs[1]};
        for (int i = 0; i < 2; ++i) {
            rcu_lazy* t = side[i];
            if (!inner(t, K_BINARY, RCU_F32) || t->op != RCU_MUL || t->rank != 4 || t->srcs[1]->numel() != 1 || t->srcs[1]->dt != RCU_F32 || t->srcs[0]->rank != 4)
                return false;
            (i ? op.scale_k : op.scale_q) = t->srcs[1];
            side[i] = t->srcs[0];
            seen.push_back(t);
        }
        rcu_lazy *q = side[0], *k = side[1];
        if (q->shape[0] != 1 || q->shape[1] != H || q->shape[2] != T || k->shape[0] != 1 || k->shape[1] != H || k->shape[3] != L || k->shape[2] != q->shape[3] ||
            v->dt != RCU_F32 || v->rank != 4 || v->shape[0] != 1 || v->shape[1] != H || v->shape[2] != L || q->shape[3] > 64 || v->shape[3] > 64)
            return false;
        op.D = (uint32_t)q->shape[3];
        op.E = (uint32_t)v->shape[3];
        op.q = strides(q, false, &seen, RCU_F32);
        op.k = strides(k, true, &seen, RCU_F32);
        op.v = strides(v, false, &seen, RCU_F32);
        for (const Heads* h : {&op.q, &op.k, &op.v})
            if (!h->base || h->offset % 4 || !aligned(h->base)) return false;
        if (!rcu_attention_f32_takes(dev, args32(op))) return false;
        op.srcs = {op.q.base, op.k.base, op.v.base, op.scale_q, op.scale_k};
        return give(root, std::move(op), seen);
    }

    // sizes and pitches; no addresses
    static Attention32Args args32(const Op& op) {
        Attention32Args a{};
        a.q = HeadRows{nullptr, op.q.head, op.q.row};
        a.k = HeadRows{nullptr, op.k.head, op.k.row};
        a.v = HeadRows{nullptr, op.v.head, op.v.row};
        a.H = (int)op.H; a.T = (int)op.T; a.L = (int)op.L; a.D = (int)op.D; a.E = (int)op.E;
        return a;
    }

    // q or k behind its slice, view, permute and rope, from the node that casts back to f16
    bool rotated(rcu_lazy* root, Op* op, std::vector<rcu_lazy*>* seen) const {
        if (root->kind != K_CAST || root->dt != RCU_F16 || root->rank != 4 || root->shape[0] != 1 || root->shape[2] < 2) return false;
        rcu_lazy* rope = root->srcs[0];
        if (!inner(rope, K_ROPE, RCU_F32)) return false;
        rcu_lazy* up = rope->srcs[0];
        if (!inner(up, K_CAST, RCU_F32) || up->srcs[0]->dt != RCU_F16) return false;
        seen->insert(seen->end(), {rope, up});
        op->H = (uint32_t)root->shape[1];
        op->T = (uint32_t)root->shape[2];
        op->D = (uint32_t)root->shape[3];
        op->q = strides(up->srcs[0], false, seen);
        op->rope.dim = rope->u[0];
        op->rope.base = rope->f[1];
        op->rope.offset = rope->u[1];
        // (rcu_rope refuses no features, and more than there are)
        return vectors(op->q) && op->D % 8 == 0 && op->rope.dim > 0 && op->rope.dim <= op->D && op->rope.dim % 16 == 0 && (uint64_t)op->T * op->D <= 0x7fffffffull;
    }

    bool heads(rcu_lazy* root) {
        Op op;
        std::vector<rcu_lazy*> seen;
        if (!rotated(root, &op, &seen)) return false;
        op.kind = HEADS;
        op.srcs = {op.q.base};
        return give(root, std::move(op), seen);
    }

    // the cache node `t` only appends: from where its source's heads come from, if these are its own
    void append(rcu_lazy* t) {
        Op op;
        op.kind = APPEND;
        rcu_lazy* x = t->srcs[1];
        std::vector<rcu_lazy*> seen;
        bool direct = false;
        if (inner(x) && x->shape[2] > 1) {
            seen.push_back(x);
            if (x->kind == K_CAST) {
                direct = rotated(x, &op, &seen);
            } else if (x->kind == K_PERMUTE && permutes(x, 0, 2, 1, 3)) {
                seen.clear();
                op.H = (uint32_t)x->shape[1];
                op.T = (uint32_t)x->shape[2];
                op.D = (uint32_t)x->shape[3];
                op.q = strides(x, false, &seen);
                direct = vectors(op.q) && op.D % 8 == 0 && (uint64_t)op.T * op.D <= 0x7fffffffull;
            }
        }
        if (direct) {
            const std::vector<rcu_lazy*> reads = {op.q.base};
            op.srcs = {t->srcs[0], op.q.base};
            if (give(t, Op(op), seen, reads)) return;
        }
        op = Op{};
        op.kind = APPEND;
        op.copied = true;
        op.srcs = {t->srcs[0], x};
        give(t, std::move(op), {}, {});
    }

    // cast(op(cast x)) of an f16 tensor: the op, null if it is another graph
    rcu_lazy* between_casts(rcu_lazy* root, int kind, std::vector<rcu_lazy*>* seen) const {
        if (root->kind != K_CAST || root->dt != RCU_F16) return nullptr;
        rcu_lazy* t = root->srcs[0];
        if (!inner(t, kind, RCU_F32)) return nullptr;
        rcu_lazy* up = t->srcs[0];
        if (!inner(up, K_CAST, RCU_F32) || up->srcs[0]->dt != RCU_F16) return nullptr;
        seen->insert(seen->end(), {t, up});
        return t;
    }

    static uint64_t rows_of(const rcu_lazy* t) { return t->numel() / t->shape[t->rank - 1]; }

    // the product `mm` (x W^T + bias in f16) as a LINEAR op, its bias's cast passed over
    bool product(const rcu_lazy* mm, bool glu, bool act, Op* op, std::vector<rcu_lazy*>* seen) const {
        if (mm->kind != K_MATMUL || mm->dt != RCU_F16 || mm->resolved() || mm->flags[0] || !mm->flags[1] || !mm->flags[2]) return false;
        rcu_lazy *w = mm->srcs[0], *x = mm->srcs[1];
        if (w->rank != 2 || x->dt != RCU_F16 || x->rank < 2) return false;
        op->kind = LINEAR;
        op->w = w;
        op->x = x;
        op->N = w->shape[0];
        op->K = w->shape[1];
        op->M = x->numel() / x->shape[x->rank - 1];
        if (x->shape[x->rank - 1] != op->K || mm->numel() != op->M * op->N || !aligned(w) || !aligned(x) || !rcu_gemm_tc_chain_takes(dev, w->dt, op->M, op->N, op->K, glu, act)) return false;
        op->srcs = {w, x};
        if (mm->srcs.size() < 3) return true;
        rcu_lazy* b = mm->srcs[2];
        if (glu || b->numel() != op->N) return false;
        if (inner(b, K_CAST, RCU_F16) && b->srcs[0]->dt == RCU_F32) {
            seen->push_back(b);
            op->bias32 = b->srcs[0];
        } else if (b->dt == RCU_F16) {
            op->bias = b;
        } else {
            return false;                // rcu_matmul refuses it
        }
        op->srcs.push_back(op->bias32 ? op->bias32 : op->bias);
        return true;
    }

    // a product whose bias is cast, one in front of an addition, or one in front of an activation between casts
    bool linear(rcu_lazy* root) {
        Op op;
        std::vector<rcu_lazy*> seen;
        if (root->kind == K_MATMUL) {
            if (!product(root, false, false, &op, &seen) || !op.bias32) return false;
        } else if (root->kind == K_BINARY && root->op == RCU_ADD && root->dt == RCU_F16) {
            for (int i = 0; i < 2 && !op.resid; ++i) {
                rcu_lazy *g = root->srcs[i], *r = root->srcs[1 - i];
                if (!inner(g, K_MATMUL, RCU_F16) || g == r || r->dt != RCU_F16 || r->rank != g->rank || root->rank != g->rank || !aligned(r)) continue;
                if (!std::equal(g->shape, g->shape + g->rank, r->shape)) continue;
                op = Op{};
                seen.assign(1, g);
                if (product(g, false, false, &op, &seen)) op.resid = r;
            }
            if (!op.resid) return false;
            op.srcs.push_back(op.resid);
        } else {
            rcu_lazy* t = between_casts(root, K_UNARY, &seen);
            if (!t || (t->op != RCU_GELU && t->op != RCU_SILU)) return false;
            rcu_lazy* g = seen[1]->srcs[0];
            if (!inner(g, K_MATMUL, RCU_F16) || !product(g, false, true, &op, &seen)) return false;
            seen.push_back(g);
            op.act = t->op;
        }
        return give(root, std::move(op), seen);
    }

    // an f32 product in front of an addition, of more than 64 tokens.  Phi-2's MLP block with the addition apart / in the epilogue, us: 65 tokens 119.2 /
    // 118.5, 128 133.4 / 133.1, Whisper-tiny's encoder of 3000 frames 563 / 545; with this rule opened 64 76.2 / 77.9, 33 74.8 / 73.0, 9 65.8 / 63.9 (not taken up:
    // small graphs then launch fewer kernels than ops, which their callers' counts would have to allow for).
    bool linear32(rcu_lazy* root) {
        if (root->op != RCU_ADD || root->dt != RCU_F32) return false;
        for (int i = 0; i < 2; ++i) {
            rcu_lazy *g = root->srcs[i], *r = root->srcs[1 - i];
            if (!inner(g, K_MATMUL, RCU_F32) || g == r || r->dt != RCU_F32 || r->rank != g->rank || root->rank != g->rank || !std::equal(g->shape, g->shape + g->rank, r->shape)) continue;
            if (g->flags[0] || !g->flags[1] || !g->flags[2]) continue;
            Op op;
            op.kind = LINEAR;
            op.full = true;
            op.w = g->srcs[0];
            op.x = g->srcs[1];
            op.resid = r;
            if (op.w->rank != 2 || (op.w->dt != RCU_F32 && op.w->dt != RCU_Q8_0F) || op.x->dt != RCU_F32 || op.x->rank < 2) continue;
            op.N = op.w->shape[0];
            op.K = op.w->shape[1];
            op.M = op.x->numel() / op.x->shape[op.x->rank - 1];
            if (op.x->shape[op.x->rank - 1] != op.K || g->numel() != op.M * op.N || !aligned(op.w) || !aligned(op.x) || op.M <= 64 || !rcu_gemm_parts_f32_takes(dev, op.M, op.N, op.K)) continue;
            op.srcs = {op.w, op.x, r};
            if (g->srcs.size() > 2) {
                op.bias = g->srcs[2];
                if (op.bias->dt != RCU_F32 || op.bias->numel() != op.N || !aligned(op.bias)) continue;      // rcu_matmul has the say
                op.srcs.push_back(op.bias);
            }
            return give(root, std::move(op), {g});
        }
        return false;
    }

    // glu of a bf16 product that nothing else reads
    bool glu_rows(rcu_lazy* root) {
        rcu_lazy* l = root->srcs[0];
        if (root->dt != RCU_BF16 || !inner(l, K_LINEAR, RCU_BF16) || l->flags[0] || l->flags[1] || l->op != RCU_ACT_NONE || l->f[0] != 1.0f) return false;
        Op op;
        op.kind = LINEAR;
        op.w = l->srcs[0];
        op.x = l->srcs[1];
        op.N = op.w->shape[0];
        op.K = op.w->shape[1];
        op.x_col = l->u[0];
        op.M = l->numel() / op.N;
        op.glu = root->op;
        const uint64_t pitch = op.x->shape[op.x->rank - 1];
        if (l->u[1] > op.N || op.w->dt != RCU_BF16 || op.x->dt != RCU_BF16 || pitch % 8 || op.x_col % 8 || !aligned(op.w) || !aligned(op.x) ||
            !rcu_gemm_tc_chain_takes(dev, RCU_BF16, op.M, op.N, op.K, true, false))
            return false;
        op.srcs = {op.w, op.x};
        return give(root, std::move(op), {l});
    }

    bool norm(rcu_lazy* root) {
        std::vector<rcu_lazy*> seen;
        rcu_lazy* t = between_casts(root, K_NORM, &seen);
        const uint64_t N = root->shape[root->rank - 1];
        if (!t || t->op == RCU_GROUP_NORM || N % 8 || N > 8192 || rows_of(root) < 2 || rows_of(root) > 0x7fffffffull) return false;
        for (size_t i = 1; i < t->srcs.size(); ++i)
            if (t->srcs[i]->dt != RCU_F32 || t->srcs[i]->numel() != N || !aligned(t->srcs[i])) return false;
        if (!aligned(seen[1]->srcs[0])) return false;
        Op op;
        op.kind = NORM;
        op.srcs = t->srcs;
        op.srcs[0] = seen[1]->srcs[0];
        return give(root, std::move(op), seen);
    }

    bool act(rcu_lazy* root) {
        std::vector<rcu_lazy*> seen;
        rcu_lazy* t = between_casts(root, K_UNARY, &seen);
        if (!t || (t->op != RCU_GELU && t->op != RCU_SILU) || root->numel() % 8 || rows_of(root) < 2 || !aligned(seen[1]->srcs[0])) return false;
        Op op;
        op.kind = ACT;
        op.srcs = {seen[1]->srcs[0]};
        return give(root, std::move(op), seen);
    }

    bool rows(rcu_lazy* root) {
        std::vector<rcu_lazy*> seen;
        rcu_lazy* sum = root;
        if (root->kind == K_CAST) {
            sum = root->srcs[0];
            if (root->dt != RCU_F16 || !inner(sum, K_BINARY, RCU_F32)) return false;
            seen.push_back(sum);
        }
        if (sum->kind != K_BINARY || sum->dt != RCU_F32 || sum->op != RCU_ADD || sum->rank != 3) return false;
        for (int i = 0; i < 2; ++i) {
            rcu_lazy *p = sum->srcs[i], *e = sum->srcs[1 - i];
            if (!inner(p, K_PERMUTE, RCU_F32) || p->rank != 3 || p->u[0] != 0 || p->u[1] != 2 || p->u[2] != 1 || p->shape[0] != 1 || p == e) continue;
            rcu_lazy* a = p->srcs[0];
            const uint64_t T = p->shape[1], C = p->shape[2];
            if (!inner(a, K_UNARY, RCU_F32) || (a->op != RCU_GELU && a->op != RCU_SILU) || T < 2 || T > 0x7fffffffull || (C + 31) / 32 > 65535) continue;
            // many pieces of 32 x 32 that are mostly empty (us apart / in one, f32: 2 x 100000 13.0 / 8.3, 2 x 1000000 37 / 58, 8 x 500000 29 / 32, 16 x 100000 13.0 / 9.0)
            const uint64_t pieces = (T + 31) / 32 * ((C + 31) / 32);
            if (pieces > 4096 && T * C < pieces * 384) continue;
            if (e->dt != RCU_F32 || e->rank < 2 || e->numel() != T * C || e->shape[e->rank - 1] != C || e->shape[e->rank - 2] != T || sum->numel() != T * C) continue;
            Op op;
            op.kind = ROWS;
            op.act = a->op;
            op.full = root->dt == RCU_F32;
            op.M = T;
            op.N = C;
            op.srcs = {a->srcs[0], e};
            seen.insert(seen.end(), {p, a});
            return give(root, std::move(op), seen);
        }
        return false;
    }

    // up * cast(silu(cast gate)), gate and up the halves of one tensor's last dimension
    bool glu(rcu_lazy* root) {
        if (root->kind != K_BINARY || root->op != RCU_MUL || root->dt != RCU_F16) return false;
        rcu_lazy *up = root->srcs[0], *a = root->srcs[1];
        if (!inner(up, K_SLICE, RCU_F16) || !inner(a, K_CAST, RCU_F16)) return false;
        std::vector<rcu_lazy*> seen{up, a};
        rcu_lazy* t = between_casts(a, K_UNARY, &seen);
        if (!t || (t->op != RCU_GELU && t->op != RCU_SILU)) return false;
        rcu_lazy* gate = seen.back()->srcs[0];
        if (!inner(gate, K_SLICE, RCU_F16) || gate->srcs[0] != up->srcs[0] || gate->rank != up->rank) return false;
        seen.push_back(gate);
        const rcu_lazy* x = up->srcs[0];
        const uint32_t r = x->rank;
        const uint64_t F = root->shape[root->rank - 1];
        if (r != up->rank || x->shape[r - 1] != 2 * F || F % 8 || F > 0x7fffffffull || gate->a[r - 1] != 0 || up->a[r - 1] != F || up->shape[r - 1] != F || gate->shape[r - 1] != F) return false;
        for (uint32_t i = 0; i + 1 < r; ++i)
            if (gate->a[i] || up->a[i] || gate->shape[i] != x->shape[i] || up->shape[i] != x->shape[i]) return false;
        if (rows_of(root) < 2 || root->numel() * 2 != x->numel() || !aligned(x)) return false;
        Op op;
        rcu_lazy* p = up->srcs[0];
        if (p->kind == K_MATMUL && !p->resolved() && p->refs.load() == 2 && !absorbed(p) && !find(p) && product(p, true, false, &op, &seen)) {       // gate and up are all that reads it
            op.glu = t->op;
            seen.push_back(p);
        } else {
            op = Op{};
            op.kind = GLU;
            op.srcs = {p};
        }
        return give(root, std::move(op), seen);
    }

    // consumers before what they consume, so that a chain is recognised from its end
    Pass(rcu_device* d, const Order& o, bool on) : dev(d), order(o), role(o.nodes.size(), kPlain) {
        if (!on) return;
        for (const rcu_lazy* t : o.nodes) {
            if (t->resolved()) continue;
            const bool first = t->kind == K_CACHE || t->kind == K_INDEX_WRITE, third = t->kind == K_LIGHTNING, fourth = t->kind == K_LATENT_APPEND || t->kind == K_KV_APPEND;
            if (!first && !third && !fourth) continue;
            const rcu_lazy* w = viewed(t->srcs[first ? 0 : third ? 2 : 3]);
            const char* begin = w->resolved() ? (const char*)w->storage->ptr : nullptr;
            written.push_back(Written{w, begin, begin ? begin + w->nbytes() : nullptr});
        }
        for (size_t i = o.nodes.size(); i-- > 0;) {
            rcu_lazy* t = o.nodes[i];
            if (t->resolved() || absorbed(t) || find(t)) continue;
            if (t->kind == K_PERMUTE) attention(t) || attention32(t);
            else if (t->kind == K_CAST) heads(t) || norm(t) || linear(t) || act(t) || rows(t);
            else if (t->kind == K_BINARY) glu(t) || linear(t) || linear32(t) || rows(t);
            else if (t->kind == K_MATMUL) linear(t);
            else if (t->kind == K_GLU) glu_rows(t);
        }
    }
};

inline const char* name_of(Kind k) {
    static const char* names[] = {"", "attention", "attention", "heads", "cache", "norm chain", "act chain", "glu chain", "linear chain", "rows chain"};
    return names[k];
}

// cos and sin of a prompt's angles, worked out once for all the layers of a resolve
struct RopeTables {
    rcu_device* dev;
    struct Entry { HeadsRope rope; uint32_t T; void* table; };
    std::vector<Entry> made;
    explicit RopeTables(rcu_device* d) : dev(d) {}
    ~RopeTables() {
        for (Entry& e : made) rcu_free(dev, e.table);          // the pool reuses blocks in stream order
    }
    rcu_status of(HeadsRope* rope, uint32_t T) {
        if (rope->dim == 0) return RCU_OK;
        for (Entry& e : made)
            if (e.T == T && e.rope.dim == rope->dim && e.rope.base == rope->base && e.rope.offset == rope->offset) {
                rope->table = e.table;
                return RCU_OK;
            }
        Entry e{*rope, T, nullptr};
        rcu_status st = rcu_alloc(dev, (uint64_t)T * rope->dim * 4, &e.table);
        if (st != RCU_OK) return st;
        made.push_back(e);
        rope->table = e.table;
        return rcu_heads_angles(dev, *rope, T, e.table);
    }
};

rcu_status run(rcu_device* dev, rcu_lazy* t, const Op& op, RopeTables* tables, void* converted) {
    HeadsRope rope = op.rope;
    if (op.kind == HEADS || (op.kind == APPEND && !op.copied)) {
        const rcu_status st = tables->of(&rope, op.T);
        if (st != RCU_OK) return st;
    }
    auto data = [](const rcu_lazy* x) { return x ? x->storage->ptr : nullptr; };
    switch (op.kind) {
        case ATTENTION: {
            AttentionArgs a{};
            a.q = op.q.rows();
            a.k = op.k.rows();
            a.v = op.v.rows();
            a.out = t->storage->ptr;
            a.H = (int)op.H; a.T = (int)op.T; a.L = (int)op.L; a.D = (int)op.D; a.E = (int)op.E;
            a.scale32[0] = (const float*)data(op.scale);
            a.scale16[0] = (const __half*)data(op.scale_q);
            a.scale16[1] = (const __half*)data(op.scale_k);
            a.mask = (const __half*)data(op.mask);
            return rcu_attention_f16(dev, a);
        }
        case ATTENTION32: {
            Attention32Args a = Pass::args32(op);
            auto at = [&](HeadRows& r, const Heads& h) { r.data = (const float*)h.base->storage->ptr + h.offset; };
            at(a.q, op.q);
            at(a.k, op.k);
            at(a.v, op.v);
            a.out = t->storage->ptr;
            a.scale[0] = (const float*)data(op.scale_q);
            a.scale[1] = (const float*)data(op.scale_k);
            return rcu_attention_f32(dev, a);
        }
        case HEADS:
            return rcu_heads_half(dev, op.q.rows(), HeadRows{t->storage->ptr, (uint64_t)op.T * op.D, op.D}, op.H, op.T, op.D, rope);
        case APPEND: {
            rcu_lazy* c = op.srcs[0];
            rcu_tensor cd = c->desc();
            if (op.copied) {
                rcu_tensor sd = op.srcs[1]->desc();
                return rcu_cache(dev, &cd, &sd, t->u[0], t->u[1], nullptr);
            }
            const uint64_t D = c->shape[3];
            return rcu_heads_half(dev, op.q.rows(), HeadRows{(char*)c->storage->ptr + t->u[1] * D * 2, c->shape[2] * D, D}, op.H, op.T, op.D, rope);
        }
        case NORM: {
            const rcu_lazy* n = t->srcs[0];
            const uint64_t N = t->shape[t->rank - 1];
            const bool bias = op.srcs.size() > 2 && n->op == RCU_LAYER_NORM;
            return rcu_norm_half(dev, n->op, data(op.srcs[0]), data(op.srcs[1]), bias ? data(op.srcs[2]) : nullptr, n->f[0], t->storage->ptr, t->numel() / N, N);
        }
        case ACT: return rcu_act_half(dev, t->srcs[0]->op, data(op.srcs[0]), t->storage->ptr, t->numel());
        case GLU: {
            const uint64_t F = t->shape[t->rank - 1];
            return rcu_glu_half(dev, t->srcs[1]->srcs[0]->op, data(op.srcs[0]), t->storage->ptr, t->numel() / F, F);
        }
        case ROWS: return rcu_act_rows(dev, op.act, (const float*)data(op.srcs[0]), (const float*)data(op.srcs[1]), t->storage->ptr, !op.full, op.M, op.N);
        case LINEAR: {
            if (op.full) {
                const void* w = converted ? converted : op.w->dt == RCU_F32 ? op.w->storage->ptr : nullptr;
                rcu_status st = w ? rcu_gemm_parts_f32_resid(dev, w, op.x->storage->ptr, data(op.bias), op.resid->storage->ptr, t->storage->ptr, op.M, op.N, op.K) : RCU_ERR_UNSUPPORTED;
                if (st != RCU_ERR_UNSUPPORTED) return st;
                rcu_tensor l = op.w->desc(), x = op.x->desc(), y = t->desc(), r = op.resid->desc(), b;
                if (converted) {
                    l.dt = RCU_F32;
                    l.data = converted;
                }
                if (op.bias) b = op.bias->desc();
                st = rcu_matmul(dev, &l, &x, op.bias ? &b : nullptr, false, true, true, &y);
                return st == RCU_OK ? rcu_binary(dev, RCU_ADD, &y, &r, &y) : st;
            }
            LinearChain c;
            c.bias = data(op.bias);
            c.bias32 = (const float*)data(op.bias32);
            c.resid = data(op.resid);
            c.op = op.act;
            c.glu = op.glu;
            c.x_pitch = op.x->shape[op.x->rank - 1];
            return rcu_gemm_tc_chain(dev, converted ? RCU_F16 : op.w->dt, converted ? converted : op.w->storage->ptr, (const char*)op.x->storage->ptr + op.x_col * 2, t->storage->ptr, op.M, op.N, op.K, c);
        }
        default: return rcu_fail(dev, RCU_ERR_UNSUPPORTED, "resolve: fused op %d", op.kind);
    }
}

}  // namespace fusion
