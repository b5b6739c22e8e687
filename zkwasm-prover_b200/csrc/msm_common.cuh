// Device helpers shared by the single and the batched MSM pipelines: point
// loads / stores and the final window combination.
#pragma once
#include "common.cuh"

namespace zk {

__device__ __forceinline__ Aff ld_aff(const Aff* p) {
    Aff a;
    a.x = ldg_elem<FqCfg>(&p->x);
    a.y = ldg_elem<FqCfg>(&p->y);
    return a;
}

__device__ __forceinline__ Xyzz ld_xyzz(const Xyzz* p) {
    Xyzz r;
    r.x = ld_elem<FqCfg>(&p->x);
    r.y = ld_elem<FqCfg>(&p->y);
    r.zz = ld_elem<FqCfg>(&p->zz);
    r.zzz = ld_elem<FqCfg>(&p->zzz);
    return r;
}

__device__ __forceinline__ void st_xyzz(Xyzz* p, const Xyzz& v) {
    st_elem<FqCfg>(&p->x, v.x);
    st_elem<FqCfg>(&p->y, v.y);
    st_elem<FqCfg>(&p->zz, v.zz);
    st_elem<FqCfg>(&p->zzz, v.zzz);
}

// ---------------------------------------------------------------------------
// Point arithmetic by quads of lanes, where the time is the latency of one
// operation: the final combination  sum_w 2^(c w) S_w  (Horner, (W - 1) c
// doublings), the trees of the bucket reduction and the merge of split buckets.
//
// Lane k of a quad holds component k of a point (X, Y, ZZ, ZZZ) and computes
// product k of the up to four independent products of a formula level; a
// level's results reach the next one's operands by shuffles inside the quad.  An
// addition takes four products of a warp, a doubling three, where one lane on
// its own takes fourteen and nine, and a warp runs eight of them side by side.
// All 32 lanes call these functions.  Coordinates lie in [0, 2p); ZZ of the
// identity is zero itself, as are its other components.  Alone on a
// sub-partition a quad addition takes 4400 clocks and a doubling 2800, a lane's
// own addition 13100 and doubling 8700 (a product is 850-900 clocks of latency).

static constexpr int COOP_THREADS = 32;

__device__ __forceinline__ int qd_lane() { return threadIdx.x & 3; }

__device__ __forceinline__ Fq qd_shfl(const Fq& v, int src) {
    Fq r;
#pragma unroll
    for (int j = 0; j < 8; j++) r.v[j] = __shfl_sync(0xffffffffu, v.v[j], src, 4);
    return r;
}

__device__ __forceinline__ Fq qd_xor2(const Fq& v) {
    Fq r;
#pragma unroll
    for (int j = 0; j < 8; j++) r.v[j] = __shfl_xor_sync(0xffffffffu, v.v[j], 2);
    return r;
}

__device__ __forceinline__ Fq qd_sel(bool c, const Fq& a, const Fq& b) {
    Fq r;
#pragma unroll
    for (int j = 0; j < 8; j++) r.v[j] = c ? a.v[j] : b.v[j];
    return r;
}

__device__ __forceinline__ Fq qd_load(const Xyzz* p) { return ld_elem<FqCfg>(reinterpret_cast<const Fq*>(p) + qd_lane()); }
__device__ __forceinline__ void qd_store(Xyzz* p, const Fq& v) {
    st_elem<FqCfg>(reinterpret_cast<Fq*>(p) + qd_lane(), fe_canon<FqCfg>(v));
}

// 2 p: dbl-2008-s-1 with (Y, 3/2 X^2) for (2 Y, 3 X^2), i.e. its result scaled
// by (1/4, 1/8, 1/4, 1/8), the same point
__device__ __forceinline__ Fq qd_dbl(const Fq& p) {
    const int k = qd_lane();
    // X^2, V = Y^2; M = 3/2 X^2
    const Fq r = fe_mul_lazy<FqCfg>(p, p);
    Fq h = r;
    limbs_half_mod<FqCfg>(h.v);
    h = fe_add_lazy<FqCfg>(r, h);
    const Fq V = qd_shfl(r, 1), M = qd_shfl(h, 0);
    // S = X V, W = Y V, ZZ3 = ZZ V, M^2
    const Fq r2 = fe_mul_lazy<FqCfg>(qd_sel(k == 3, M, p), qd_sel(k == 3, M, V));
    const Fq mm = qd_shfl(r2, 3), W = qd_shfl(r2, 1);
    const Fq s2 = fe_add_lazy<FqCfg>(r2, r2);
    const Fq x3 = fe_sub_lazy<FqCfg>(mm, s2);
    const Fq t = fe_sub_lazy<FqCfg>(fe_add_lazy<FqCfg>(s2, r2), mm);  // S - X3
    // M (S - X3), Y W, -, ZZZ W
    const Fq r3 = fe_mul_lazy<FqCfg>(qd_sel(k == 0, M, p), qd_sel(k == 0, t, W));
    const Fq y3 = fe_sub_lazy<FqCfg>(qd_shfl(r3, 0), r3);
    return qd_sel(k < 2, qd_sel(k == 0, x3, y3), qd_sel(k == 2, r2, r3));
}

// p + q (add-2008-s)
__device__ __forceinline__ Fq qd_add(const Fq& p, const Fq& q) {
    const int k = qd_lane();
    const int zz = (threadIdx.x & 28) + 2;  // this quad's ZZ lane
    const bool idp = (__ballot_sync(0xffffffffu, fe_is_zero<FqCfg>(p)) >> zz) & 1u;
    const bool idq = (__ballot_sync(0xffffffffu, fe_is_zero<FqCfg>(q)) >> zz) & 1u;
    // U1 = X1 ZZ2, S1 = Y1 ZZZ2, U2 = ZZ1 X2, S2 = ZZZ1 Y2
    const Fq r = cmul_lazy(p, qd_xor2(q));
    const Fq d = fe_sub_lazy<FqCfg>(qd_xor2(r), r);  // P = U2 - U1, R = S2 - S1 in lanes 0, 1
    const unsigned zd = __ballot_sync(0xffffffffu, fe_is_zero<FqCfg>(fe_canon<FqCfg>(d))) >> (threadIdx.x & 28);
    // P^2, R^2, ZZ1 ZZ2, ZZZ1 ZZZ2
    const Fq r2 = cmul_lazy(qd_sel(k < 2, d, p), qd_sel(k < 2, d, q));
    const Fq PP = qd_shfl(r2, 0), U1 = qd_shfl(r, 0);
    // PPP = P PP, Q = U1 PP, ZZ3 = ZZ1 ZZ2 PP
    const Fq r3 = cmul_lazy(qd_sel(k == 0, d, qd_sel(k == 1, U1, r2)), PP);
    const Fq PPP = qd_shfl(r3, 0), S1 = qd_shfl(r, 1);
    // lane 1 holds R^2 and Q
    const Fq x3 = fe_sub_lazy<FqCfg>(fe_sub_lazy<FqCfg>(r2, PPP), fe_add_lazy<FqCfg>(r3, r3));
    const Fq t = fe_sub_lazy<FqCfg>(r3, x3);
    // S1 PPP, R (Q - X3), -, ZZZ3 = ZZZ1 ZZZ2 PPP
    const Fq r4 = cmul_lazy(qd_sel(k == 0, S1, qd_sel(k == 1, d, r2)), qd_sel(k == 1, t, PPP));
    const Fq y3 = fe_sub_lazy<FqCfg>(r4, qd_shfl(r4, 0));
    Fq res = qd_sel(k < 2, qd_sel(k == 0, qd_shfl(x3, 1), y3), qd_sel(k == 2, r3, r4));
    const bool same_x = (zd & 1u) && !idp && !idq;
    if (__any_sync(0xffffffffu, same_x)) {
        const Fq dd = qd_dbl(p);
        if (same_x) res = qd_sel(zd & 2u, dd, fe_zero<FqCfg>());
    }
    return qd_sel(idq, p, qd_sel(idp, q, res));
}

// the point with canonical coordinates, in every lane
__device__ __forceinline__ Xyzz qd_point(const Fq& p) {
    Xyzz r;
    r.x = qd_shfl(p, 0);
    r.y = qd_shfl(p, 1);
    r.zz = qd_shfl(p, 2);
    r.zzz = qd_shfl(p, 3);
    return xyzz_canon(r);
}

// Horner over the W window sums win[0..W) of one MSM by one warp (its quads
// all compute the same)
__device__ __forceinline__ Jac coop_horner(const Xyzz* win, int W, int c) {
    Fq acc = fe_zero<FqCfg>();
    int w = W - 1;
    if (w >= 0) acc = qd_load(win + w);
    // small scalars leave the top windows empty
    while (w > 0 && __all_sync(0xffffffffu, fe_is_zero<FqCfg>(acc))) acc = qd_load(win + --w);
    while (--w >= 0) {
        const Fq next = qd_load(win + w);
#pragma unroll 1
        for (int i = 0; i < c; i++) acc = qd_dbl(acc);
        acc = qd_add(acc, next);
    }
    return xyzz_to_jac(qd_point(acc));
}

// ---------------------------------------------------------------------------
// Bucket reduction  sum_b (b + 1) B_b  of a set of B buckets, in G = B / seg
// segments (seg and G powers of two, G <= RED_MAX_G).
//
// A thread sums segment g by running sums: S_g = sum_j (j + 1) B_{g seg + j}
// and T_g = sum_j B_{g seg + j}; the set's sum is then
//     sum_g S_g + seg * sum_g g T_g,   sum_g g T_g = sum_k 2^k V_k,
// with V_k the sum of the T_g whose g has bit k set.  All V_k come out of one
// pairwise tree over the T_g: where a node joins its halves, V_k of the node is
// the sum of its halves' V_k, and the V of the bit that tells the halves apart
// is the right half's T.  So no thread multiplies its T by its segment's
// number (about 1.5 log2 B additions' worth of doublings and additions each,
// which was most of the reduction's work where segments are short), and what
// is left is one short Horner chain a set.
//
// Stages: (1) a block of RED_T threads sums RED_T segments and runs the tree
// over each group of GS = min(G, RED_T) of them; (2) where a set has H = G / GS
// > 1 groups, one block for each of its nine planes (S, V_0..V_6, T) sums the
// plane over the groups, the T plane by the same tree; (3) one block a set runs
// the Horner chain.  A set's points lie plane by plane from its first slot
// (plane p of group h at p H + h), stage 2's results after them.
static constexpr uint32_t RED_T = 128;
static constexpr uint32_t RED_LG = 7;
static constexpr uint32_t RED_MAX_G = RED_T * RED_T;
static constexpr uint32_t RED_PLANES = RED_LG + 2;

// Trees over the groups of 2^lg leaves of Tp and Sp (either may be null), RED_T
// leaves each, one addition a quad; every thread of the block calls it after a
// barrier.  Node base of level l holds T at Tp[base], V_k at Tp[base + 2^k]
// (k < l) and S at Sp[base].
__device__ __forceinline__ void red_tree(Xyzz* Tp, Xyzz* Sp, uint32_t lg) {
    const uint32_t quad = threadIdx.x >> 2;
#pragma unroll 1
    for (uint32_t l = 1; l <= lg; l++) {
        // additions: row r of the level's nodes; row 0 is S, row 1 T, row 2 + k V_k
        const uint32_t nodes = RED_T >> l, first = Sp ? 0u : nodes, last = Tp ? nodes * (l + 1) : nodes;
#pragma unroll 1
        for (uint32_t a0 = first; a0 < last; a0 += RED_T / 4) {
            const uint32_t a = a0 + quad, r = a >> (RED_LG - l), base = (a & (nodes - 1)) << l;
            Xyzz* dst = r == 0 ? Sp + base : Tp + base + (r >= 2 ? 1u << (r - 2) : 0u);
            const bool live = a < last;
            Fq p = fe_zero<FqCfg>(), q = p;
            if (live) {
                p = reinterpret_cast<const Fq*>(dst)[qd_lane()];
                q = reinterpret_cast<const Fq*>(dst + (1u << (l - 1)))[qd_lane()];
            }
            // skipped where no quad of the warp has two points (an identity's
            // components are all zero): empty buckets, short and sparse columns
            const bool zq = fe_is_zero<FqCfg>(q);
            p = __all_sync(0xffffffffu, zq || fe_is_zero<FqCfg>(p)) ? qd_sel(zq, p, q) : qd_add(p, q);
            if (live) reinterpret_cast<Fq*>(dst)[qd_lane()] = p;
        }
        __syncthreads();
    }
}

// stage 1, one thread's segment: buckets key0 .. key0 + seg - 1 (empty ones,
// offset[k] == offset[k + 1], hold nothing)
__device__ __forceinline__ void red_segment(const Xyzz* buckets, const uint32_t* offset, uint32_t key0, uint32_t seg,
                                            Xyzz& S, Xyzz& T) {
    S = T = xyzz_identity();
    for (uint32_t j = seg; j-- > 0;) {
        const uint32_t key = key0 + j;
        if (offset[key + 1] != offset[key]) T = xyzz_add(T, ld_xyzz(buckets + key));
        S = xyzz_add(S, T);
    }
}

// stage 1, the block's part: S, T of thread t (identity past the end); the
// thread at the head of a group writes nothing but the group's planes, spread
// over the group's first threads.  out: the set's first slot, h: the group.
__device__ __forceinline__ void red_groups(Xyzz* Tp, Xyzz* Sp, const Xyzz& S, const Xyzz& T, uint32_t G, bool live,
                                           Xyzz* out, uint32_t h) {
    Tp[threadIdx.x] = T;
    Sp[threadIdx.x] = S;
    __syncthreads();
    const uint32_t GS = G < RED_T ? G : RED_T, lg = 31u - (uint32_t)__clz((int)GS), H = G / GS;
    red_tree(Tp, Sp, lg);
    const uint32_t p = threadIdx.x & (GS - 1), base = threadIdx.x - p;
    const uint32_t planes = lg + 1 + (H > 1 ? 1u : 0u);
    if (live && p < planes) {
        const Xyzz v = p == 0 ? Sp[base] : Tp[base + (p <= lg ? 1u << (p - 1) : 0u)];
        st_xyzz(out + p * H + h, xyzz_canon(v));
    }
}

// stage 2: plane p of a set of H > 1 groups (H <= RED_T)
__device__ __forceinline__ void red_plane(Xyzz* sm, Xyzz* set, uint32_t H, uint32_t p) {
    const uint32_t i = threadIdx.x, lg = 31u - (uint32_t)__clz((int)H);
    sm[i] = i < H ? ld_xyzz(set + p * H + i) : xyzz_identity();
    __syncthreads();
    const bool t_plane = p == RED_PLANES - 1;
    red_tree(t_plane ? sm : nullptr, t_plane ? nullptr : sm, lg);
    Xyzz* out = set + RED_PLANES * H;
    if (!t_plane) {
        if (i == 0) st_xyzz(out + p, xyzz_canon(sm[0]));
    } else if (i < lg) {
        st_xyzz(out + p + i, xyzz_canon(sm[1u << i]));
    }
}

// stage 3 by one warp: the set's sum, component qd_lane() in every quad
__device__ __forceinline__ Fq red_horner(const Xyzz* set, uint32_t G, uint32_t seg) {
    const uint32_t H = G > RED_T ? G / RED_T : 1u;
    const Xyzz* v = H > 1 ? set + RED_PLANES * H : set;
    Fq acc = fe_zero<FqCfg>();
    // the bits of the segment number from the top, seg's doublings, then S;
    // leading identities (an empty set has only those) cost nothing
    uint32_t k = 31u - (uint32_t)__clz((int)G), s = seg;
    bool some = false;
#pragma unroll 1
    while (s) {
        const bool term = k > 0 || s == 1;
        if (some) {
            if (k > 0 || s > 1) acc = qd_dbl(acc);
            if (term) acc = qd_add(acc, qd_load(v + k));
        } else if (term) {
            acc = qd_load(v + k);
            some = !__all_sync(0xffffffffu, fe_is_zero<FqCfg>(acc));
        }
        if (k > 0)
            k--;
        else
            s >>= 1;
    }
    return acc;
}

}  // namespace zk
