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
// Final combination  sum_w 2^(c w) S_w  (Horner, (W - 1) c doublings).
//
// It is one dependent chain, so its time is the latency of the products on
// the chain.  One warp's Fq product is bound by the multiply pipe of its SM
// sub-partition, so a thread cannot overlap two products; instead a CTA of
// four warps (one per sub-partition) evaluates up to four independent products
// of a formula at once: lane 0 of warp k computes product k, the results meet
// in shared memory, and every thread keeps the whole point in registers and
// does the additions itself.  A doubling (6M + 3S) becomes three product
// levels, an addition (12M + 2S) four.

static constexpr int COOP_THREADS = 128;

struct Coop {
    Fq* buf;  // shared, 2 x 4 elements (double-buffered result slots)
    int par;
};

// r_k = a_k * b_k for k < cnt, all threads receive every result
template <int CNT>
__device__ __forceinline__ void coop_mul(Coop& co, const Fq& a0, const Fq& b0, const Fq& a1, const Fq& b1,
                                         const Fq& a2, const Fq& b2, const Fq& a3, const Fq& b3, Fq& r0, Fq& r1,
                                         Fq& r2, Fq& r3) {
    const int wp = threadIdx.x >> 5;
    Fq* slot = co.buf + 4 * co.par;
    if ((threadIdx.x & 31) == 0 && wp < CNT) {
        const Fq a = wp == 0 ? a0 : wp == 1 ? a1 : wp == 2 ? a2 : a3;
        const Fq b = wp == 0 ? b0 : wp == 1 ? b1 : wp == 2 ? b2 : b3;
        slot[wp] = fe_mul<FqCfg>(a, b);
    }
    __syncthreads();
    r0 = slot[0];
    if (CNT > 1) r1 = slot[1];
    if (CNT > 2) r2 = slot[2];
    if (CNT > 3) r3 = slot[3];
    // the next call writes the other slot set; this one is rewritten only
    // after every thread has passed the next barrier, i.e. read these results
    co.par ^= 1;
}

// 2 * p, dbl-2008-s-1 in three product levels
__device__ __forceinline__ Xyzz coop_dbl(Coop& co, const Xyzz& p) {
    if (xyzz_is_id(p)) return p;
    Fq d = fe_zero<FqCfg>();
    const Fq u = fe_dbl<FqCfg>(p.y);
    Fq v, xx;
    coop_mul<2>(co, u, u, p.x, p.x, d, d, d, d, v, xx, d, d);
    const Fq mm = fe_add<FqCfg>(fe_dbl<FqCfg>(xx), xx);
    Fq w, s, m2, zz;
    coop_mul<4>(co, u, v, p.x, v, mm, mm, v, p.zz, w, s, m2, zz);
    Xyzz r;
    r.x = fe_sub<FqCfg>(fe_sub<FqCfg>(m2, s), s);
    const Fq t = fe_sub<FqCfg>(s, r.x);
    Fq zzz, wy, mt;
    coop_mul<3>(co, w, p.zzz, w, p.y, mm, t, d, d, zzz, wy, mt, d);
    r.y = fe_sub<FqCfg>(mt, wy);
    r.zz = zz;
    r.zzz = zzz;
    return r;
}

// p + q, add-2008-s in four product levels
__device__ __forceinline__ Xyzz coop_add(Coop& co, const Xyzz& p, const Xyzz& q) {
    if (xyzz_is_id(p)) return q;
    if (xyzz_is_id(q)) return p;
    Fq d = fe_zero<FqCfg>();
    Fq u1, u2, s1, s2;
    coop_mul<4>(co, p.x, q.zz, q.x, p.zz, p.y, q.zzz, q.y, p.zzz, u1, u2, s1, s2);
    const Fq P = fe_sub<FqCfg>(u2, u1);
    const Fq R = fe_sub<FqCfg>(s2, s1);
    if (fe_is_zero<FqCfg>(P)) {
        if (fe_is_zero<FqCfg>(R)) return coop_dbl(co, p);
        return xyzz_identity();
    }
    Fq pp, zzp, zzzp, rr;
    coop_mul<4>(co, P, P, p.zz, q.zz, p.zzz, q.zzz, R, R, pp, zzp, zzzp, rr);
    Fq ppp, qq, zz;
    coop_mul<3>(co, P, pp, u1, pp, zzp, pp, d, d, ppp, qq, zz, d);
    Xyzz r;
    r.x = fe_sub<FqCfg>(fe_sub<FqCfg>(fe_sub<FqCfg>(rr, ppp), qq), qq);
    const Fq t = fe_sub<FqCfg>(qq, r.x);
    Fq zzz, sp, rt;
    coop_mul<3>(co, zzzp, ppp, s1, ppp, R, t, d, d, zzz, sp, rt, d);
    r.y = fe_sub<FqCfg>(rt, sp);
    r.zz = zz;
    r.zzz = zzz;
    return r;
}

// XYZZ -> Jacobian (X ZZ^2, Y ZZ^3, ZZZ); identity -> (0, 1, 0)
__device__ __forceinline__ Jac coop_to_jac(Coop& co, const Xyzz& p) {
    Jac r;
    if (xyzz_is_id(p)) {
        r.x = fe_zero<FqCfg>();
        r.y = fe_one<FqCfg>();
        r.z = fe_zero<FqCfg>();
        return r;
    }
    Fq d = fe_zero<FqCfg>(), zz2, zz3;
    coop_mul<1>(co, p.zz, p.zz, d, d, d, d, d, d, zz2, d, d, d);
    coop_mul<2>(co, zz2, p.zz, p.x, zz2, d, d, d, d, zz3, r.x, d, d);
    coop_mul<1>(co, p.y, zz3, d, d, d, d, d, d, r.y, d, d, d);
    r.z = p.zzz;
    return r;
}

// Horner over the W window sums win[0..W) of one MSM by the whole CTA
// (COOP_THREADS threads); every thread returns the Jacobian result.
__device__ __forceinline__ Jac coop_horner(Fq* sh_buf, const Xyzz* win, int W, int c) {
    Coop co{sh_buf, 0};
    Xyzz acc = W > 0 ? ld_xyzz(win + W - 1) : xyzz_identity();
    for (int w = W - 2; w >= 0; w--) {
        for (int i = 0; i < c; i++) acc = coop_dbl(co, acc);
        acc = coop_add(co, acc, ld_xyzz(win + w));
    }
    return coop_to_jac(co, acc);
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
// is left is one short Horner chain a set.  Eight MSMs of 2^15 points (2^14
// buckets each) reduce in 230 us against 700, one of 100003 points in 167
// against 234 (ncu).
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

// Trees over the first 2^lg-leaf groups of Tp and Sp (either may be null),
// RED_T leaves each; every thread of the block calls it after a barrier.  Node
// base of level l holds T at Tp[base], V_k at Tp[base + 2^k] (k < l) and S at
// Sp[base].
__device__ __forceinline__ void red_tree(Xyzz* Tp, Xyzz* Sp, uint32_t lg) {
    for (uint32_t l = 1; l <= lg; l++) {
        // one addition a thread: at most RED_T of them on every level
        const uint32_t nodes = RED_T >> l, base = (threadIdx.x & (nodes - 1)) << l;
        const uint32_t r = threadIdx.x >> (RED_LG - l);
        Xyzz* dst = nullptr;
        if (r == 0)
            dst = Sp ? Sp + base : nullptr;
        else if (r <= l)
            dst = Tp ? Tp + base + (r >= 2 ? 1u << (r - 2) : 0u) : nullptr;
        if (dst) *dst = xyzz_add(*dst, dst[1u << (l - 1)]);
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
        st_xyzz(out + p * H + h, v);
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
        if (i == 0) st_xyzz(out + p, sm[0]);
    } else if (i < lg) {
        st_xyzz(out + p + i, sm[1u << i]);
    }
}

// stage 3 by COOP_THREADS threads: the set's sum
__device__ __forceinline__ Xyzz red_horner(Fq* sh_buf, const Xyzz* set, uint32_t G, uint32_t seg) {
    const uint32_t H = G > RED_T ? G / RED_T : 1u;
    const Xyzz* v = H > 1 ? set + RED_PLANES * H : set;
    Coop co{sh_buf, 0};
    Xyzz acc = xyzz_identity();
    for (uint32_t k = 31u - (uint32_t)__clz((int)G); k > 0; k--) {
        acc = coop_dbl(co, acc);
        acc = coop_add(co, acc, ld_xyzz(v + k));
    }
    for (uint32_t s = seg; s > 1; s >>= 1) acc = coop_dbl(co, acc);
    return coop_add(co, acc, ld_xyzz(v));
}

}  // namespace zk
