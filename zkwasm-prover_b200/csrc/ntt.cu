// Radix-2^k NTT for BN254 Fr on sm_100a.
//
// A transform of size n = 2^log_n is a sequence of global passes (Stockham
// autosort, natural order in and out).  Pass t has radix R_t = 2^LOGR and
// P_t = R_1 * ... * R_{t-1}.  Work item q in [0, n/R_t) with J = q mod P_t and
// Q = q / P_t:
//     reads   x[q + (n/R_t) * i]                       i < R_t
//     y_j   = sum_i x_i w_{P_t R_t}^{J i} w_{R_t}^{ij}  (in shared memory)
//     writes  dst[J + P_t*j + P_t*R_t*Q] = y_j
// so the final pass leaves X[j] = sum_i x_i w_n^{ij} in natural order.  Inside a
// CTA the radix-R_t DFT is itself a Stockham sequence of radix-8 (then 4 or 2)
// sub-stages held in registers, exchanging through shared memory, each of the
// same form with P_s = 8^s: input i of an item is multiplied by
// w_{P R}^{J i} over the indexes of pass and sub-stage together, then a DFT of
// eight follows.  Twiddles come before the DFT (decimation in time), so that
//   - the first sub-stage of the first pass has none;
//   - a factor common to all inputs (the scale n^-1) costs one product per
//     eight elements: it goes into the eight factors of an item's first
//     sub-stage, where input 0 otherwise has none;
//   - in the fused extension a coset shift s (X[j] = sum_k x_k s^k w^{jk}) only
//     changes factors that are multiplied by anyway: see ntt_coset_table_kernel.
//
// Twiddles come from the natural table w^i (i < n) that expand_omega_buffer
// builds; a sub-stage twiddle w_R^e is entry e * (n/R).
//
// The same pass kernel serves the coset extension: an optional per-input
// multiplier table (the coset twist s^k or any other factors, applied in the
// first pass, whose first sub-stage has no twiddles: the products an element
// are the same as with the shift in the sub-stages' factors),
// an optional output scale (n^-1 for the inverse transform) and an output
// index map pos -> (pos << out_shift) + z * out_off_z that interleaves the
// 2^e sub-transforms of an extended domain.
//
// Reference behaviour replaced: cuda/bn254.cu:1357-1428 (ntt), 294-418
// (merge_ntt_kernel), 421-494 (_ntt_core).
#include "common.cuh"
#include "kernels.h"

namespace zk {

// Every Fr product of the pass kernels goes through one out-of-line function:
// inlined, the ~30 product sites of a pass (each ~350 instructions) overflow
// the instruction cache and warps stall on instruction fetch.
//
// Inside a pass, values are kept lazily reduced in [0, 2r): the products skip
// their final conditional subtraction (nt_mulz) and the butterflies add and
// subtract modulo 2r; every value leaves a pass canonical (fe_canon at the
// last sub-stage), so buffers in global memory always hold canonical values.
#if defined(ZK_NTT_INLINE_MUL)
__device__ __forceinline__ Fr nt_mul(const Fr& a, const Fr& b) { return fe_mul<FrCfg>(a, b); }
__device__ __forceinline__ Fr nt_mulz(const Fr& a, const Fr& b) { return fe_mul_lazy<FrCfg>(a, b); }
__device__ __forceinline__ Fr nt_shoup(const Fr& a, const Fr& w, const Fr& wp) {
    return fe_mul_shoup<FrCfg>(a, w, wp);
}
#else
__device__ __noinline__ Fr nt_mul(const Fr a, const Fr b) { return fe_mul<FrCfg>(a, b); }
__device__ __noinline__ Fr nt_mulz(const Fr a, const Fr b) { return fe_mul_lazy<FrCfg>(a, b); }
__device__ __noinline__ Fr nt_shoup(const Fr a, const Fr w, const Fr wp) { return fe_mul_shoup<FrCfg>(a, w, wp); }
#endif

// Two independent products in one call, so the scheduler can interleave their
// carry chains.
struct Fr2 {
    Fr a, b;
};
#if defined(ZK_NTT_INLINE_MUL)
#define ZK_NTMUL __device__ __forceinline__
#else
#define ZK_NTMUL __device__ __noinline__
#endif
ZK_NTMUL Fr2 nt_mulz2(const Fr a0, const Fr w0, const Fr a1, const Fr w1) {
    return {fe_mul_lazy<FrCfg>(a0, w0), fe_mul_lazy<FrCfg>(a1, w1)};
}
ZK_NTMUL Fr2 nt_shoup2(const Fr a0, const Fr w0, const Fr p0, const Fr a1, const Fr w1, const Fr p1) {
    return {fe_mul_shoup<FrCfg>(a0, w0, p0), fe_mul_shoup<FrCfg>(a1, w1, p1)};
}
#undef ZK_NTMUL

// Multiplier tables (twiddles, twists, scales) come in two layouts.
// TwM: one Montgomery-form element per entry, multiplied with nt_mulz.
// TwS: the pair (w, w') per entry, w canonical and w' = floor(w 2^256 / r),
// multiplied with nt_shoup (207 multiply-adds instead of 264; both results
// lie in [0, 2r)).  Every product of the pass kernels is by a table entry.
struct TwM {
    struct K {
        Fr w;
    };
    static __device__ __forceinline__ K ld(const Fr* t, size_t i) { return {ldg_elem<FrCfg>(t + i)}; }
    static __device__ __forceinline__ Fr mul(const Fr& v, const K& k) { return nt_mulz(v, k.w); }
    static __device__ __forceinline__ Fr2 mul2(const Fr& v0, const K& k0, const Fr& v1, const K& k1) {
        return nt_mulz2(v0, k0.w, v1, k1.w);
    }
    static __host__ __device__ __forceinline__ const Fr* off(const Fr* t, size_t i) { return t + i; }
    static constexpr int EW = 1;  // elements an entry
    // the entry's value (in this layout's form) and the entry of a value
    static __device__ __forceinline__ K of(const Fr& v) { return {v}; }
    static __device__ __forceinline__ K prod(const K& a, const K& b) { return {nt_mul(a.w, b.w)}; }
    static __device__ __forceinline__ K sm(const Fr* t) { return {t[0]}; }
    static __device__ __forceinline__ void put(Fr* t, const K& k) { t[0] = k.w; }
};
struct TwS {
    struct K {
        Fr w, wp;
    };
    static __device__ __forceinline__ K ld(const Fr* t, size_t i) {
        return {ldg_elem<FrCfg>(t + 2 * i), ldg_elem<FrCfg>(t + 2 * i + 1)};
    }
    static __device__ __forceinline__ Fr mul(const Fr& v, const K& k) { return nt_shoup(v, k.w, k.wp); }
    static __device__ __forceinline__ Fr2 mul2(const Fr& v0, const K& k0, const Fr& v1, const K& k1) {
        return nt_shoup2(v0, k0.w, k0.wp, v1, k1.w, k1.wp);
    }
    static __host__ __device__ __forceinline__ const Fr* off(const Fr* t, size_t i) { return t + 2 * i; }
    static constexpr int EW = 2;
    static __device__ __forceinline__ K of(const Fr& v) {
        return {v, fe_shoup_companion<FrCfg>(fe_to_mont<FrCfg>(v))};
    }
    static __device__ __forceinline__ K prod(const K& a, const K& b) {
        return of(fe_canon<FrCfg>(nt_shoup(a.w, b.w, b.wp)));
    }
    static __device__ __forceinline__ K sm(const Fr* t) { return {t[0], t[1]}; }
    static __device__ __forceinline__ void put(Fr* t, const K& k) {
        t[0] = k.w;
        t[1] = k.wp;
    }
};


// ---------------------------------------------------------------- small DFTs

__device__ __forceinline__ void dft2(Fr& a, Fr& b) {
    Fr t = fe_add_lazy<FrCfg>(a, b);
    b = fe_sub_lazy<FrCfg>(a, b);
    a = t;
}

// The factors of a DFT of eight, kept in shared memory: w4 = w_8^2,
// cu = (w_8 + w_8^-1) / 2 and su = (w_8 - w_8^-1) / 2 (w_8^-1 = -w_8^3).
template <class TW>
struct DftK {
    Fr k[3 * TW::EW];
    __device__ __forceinline__ typename TW::K w4() const { return TW::sm(k); }
    __device__ __forceinline__ typename TW::K cu() const { return TW::sm(k + TW::EW); }
    __device__ __forceinline__ typename TW::K su() const { return TW::sm(k + 2 * TW::EW); }
    // Made by threads 0 to 2 of a block in two steps, the loads before the block's
    // tile is read and the rest after, so that one wait covers both.
    // tw: the table of w_n, n = 2^log_n >= 8
    struct Raw {
        typename TW::K a;
        Fr b;
    };
    static __device__ __forceinline__ Raw fetch(int i, const Fr* tw, int log_n) {
        Raw r;
        if (i < 3) {
            r.a = TW::ld(tw, (size_t)1 << (log_n - (i ? 3 : 2)));
            r.b = TW::ld(tw, (size_t)3 << (log_n - 3)).w;
        }
        return r;
    }
    __device__ __forceinline__ void put(int i, const Raw& r) {
        if (i >= 3) return;
        typename TW::K f = r.a;
        if (i) {
            Fr h = i == 1 ? fe_sub<FrCfg>(r.a.w, r.b) : fe_add<FrCfg>(r.a.w, r.b);
            limbs_half_mod<FrCfg>(h.v);
            f = TW::of(h);
        }
        TW::put(k + i * TW::EW, f);
    }
    __device__ __forceinline__ void init(const Fr* tw, int log_n) {
        for (int i = threadIdx.x; i < 3; i += blockDim.x) put(i, fetch(i, tw, log_n));
    }
};

// DFT of eight by Winograd's short algorithm (S. Winograd, "On computing the
// discrete Fourier transform", 1978): four products, independent of each other
// (w4 twice, cu, su), where the radix-2 form takes five in two levels.  In and
// out in natural order up to dft8_slot: y_j ends in v[dft8_slot(j)].
template <class TW>
__device__ __forceinline__ void dft8(Fr v[8], const DftK<TW>& c) {
    dft2(v[0], v[4]);
    dft2(v[2], v[6]);
    dft2(v[1], v[5]);
    dft2(v[3], v[7]);
    dft2(v[5], v[7]);  // v5: sum (su), v7: difference (cu)
    dft2(v[1], v[3]);
    if constexpr (TW::EW == 2) {
        v[5] = TW::mul(v[5], c.su());
        v[7] = TW::mul(v[7], c.cu());
        v[3] = TW::mul(v[3], c.w4());
        v[6] = TW::mul(v[6], c.w4());
    } else {
        const Fr2 a = TW::mul2(v[5], c.su(), v[7], c.cu());
        v[5] = a.a;
        v[7] = a.b;
        const Fr2 b = TW::mul2(v[3], c.w4(), v[6], c.w4());
        v[3] = b.a;
        v[6] = b.b;
    }
    dft2(v[0], v[2]);
    dft2(v[0], v[1]);
    dft2(v[2], v[3]);
    dft2(v[4], v[7]);
    dft2(v[5], v[6]);
    dft2(v[4], v[5]);
    dft2(v[7], v[6]);
}
__device__ __forceinline__ constexpr int dft8_slot(int j) {
    return j == 0 ? 0 : j == 1 ? 4 : j == 2 ? 2 : j == 3 ? 7 : j == 4 ? 1 : j == 5 ? 6 : j == 6 ? 3 : 5;
}

// v[0..3] -> y[k]: y0=v0, y1=v2, y2=v1, y3=v3
template <class TW>
__device__ __forceinline__ void dft4_dif(Fr& v0, Fr& v1, Fr& v2, Fr& v3, const typename TW::K& w4) {
    dft2(v0, v2);
    dft2(v1, v3);
    v3 = TW::mul(v3, w4);
    dft2(v0, v1);
    dft2(v2, v3);
}

// Where the factors of an item's sub-stages come from: the table of w_n at
// (i J_full) n / (P R_s) for item index J_full = J + P Jl, or ctab, the fused
// extension's table of a coset's first pass (ntt_coset_table_kernel).
struct StageTw {
    const Fr* tw;
    const Fr* ctab;
    int log_n, log_p;
    uint32_t J;  // the item's index in the products of earlier passes
};

// factor of input i of local item Jl in a sub-stage of radix 2^LR after P_s = 2^log_ps
template <int LR, class TW>
__device__ __forceinline__ typename TW::K stage_factor(const StageTw& t, uint32_t Jl, int log_ps, uint32_t i) {
    if (t.ctab) return TW::ld(t.ctab, ((((size_t)1 << log_ps) + Jl) << LR) + i);
    return TW::ld(t.tw, (size_t)(i * (t.J + (Jl << t.log_p))) << (t.log_n - t.log_p - log_ps - LR));
}

// radix-8 sub-stage over one DFT of size R in shared memory, v its inputs
// (already multiplied by their factors) in registers
template <class TW>
__device__ __forceinline__ void stage8_finish(Fr* x, int u, int log_ps, bool last, Fr v[8], const DftK<TW>& dk) {
    dft8<TW>(v, dk);
    const int J = u & ((1 << log_ps) - 1);
    const int ilo = u >> log_ps;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const Fr y = v[dft8_slot(j)];
        sm_st(x, J + (j << log_ps) + (ilo << (log_ps + 3)), last ? fe_canon<FrCfg>(y) : y);
    }
    __syncthreads();
}

// inputs 1..7 of a sub-stage by their factors
template <class TW>
__device__ __forceinline__ void stage8_twiddle(Fr v[8], const StageTw& t, uint32_t Jl, int log_ps) {
    if (!t.ctab && t.J + (Jl << t.log_p) == 0) return;
    if constexpr (TW::EW == 2) {
        // one at a time: two pairs of factors beside eight elements would spill
#pragma unroll
        for (uint32_t i = 1; i < 8; i++) v[i] = TW::mul(v[i], stage_factor<3, TW>(t, Jl, log_ps, i));
    } else {
#pragma unroll
        for (uint32_t i = 1; i < 7; i += 2) {
            const Fr2 m = TW::mul2(v[i], stage_factor<3, TW>(t, Jl, log_ps, i), v[i + 1],
                                   stage_factor<3, TW>(t, Jl, log_ps, i + 1));
            v[i] = m.a;
            v[i + 1] = m.b;
        }
        v[7] = TW::mul(v[7], stage_factor<3, TW>(t, Jl, log_ps, 7));
    }
}

// all eight inputs by k[0..7] (shared memory)
template <class TW>
__device__ __forceinline__ void stage8_scale(Fr v[8], const Fr* k) {
    if constexpr (TW::EW == 2) {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = TW::mul(v[i], TW::sm(k + i * TW::EW));
    } else {
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            const Fr2 m = TW::mul2(v[i], TW::sm(k + i * TW::EW), v[i + 1], TW::sm(k + (i + 1) * TW::EW));
            v[i] = m.a;
            v[i + 1] = m.b;
        }
    }
}

template <int LOGR, class TW>
__device__ __forceinline__ void stage8_load(Fr v[8], Fr* x, int u) {
    constexpr int S = (1 << LOGR) / 8;
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = sm_ld(x, u + S * i);
    __syncthreads();
}

// final radix-4 sub-stage (two items per thread), P_s = R / 4
template <int LOGR, class TW>
__device__ __forceinline__ void stage4_last(Fr* x, int lt, const StageTw& t, const DftK<TW>& dk) {
    constexpr int R = 1 << LOGR;
    constexpr int S = R / 4;  // items and read stride
    constexpr int TH = R / 8;
    // a thread rewrites only its own slots u + S j
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        const uint32_t u = lt + k * TH;
        Fr v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = sm_ld(x, u + S * i);
        const Fr2 m = TW::mul2(v[1], stage_factor<2, TW>(t, u, LOGR - 2, 1), v[2],
                               stage_factor<2, TW>(t, u, LOGR - 2, 2));
        v[1] = m.a;
        v[2] = m.b;
        v[3] = TW::mul(v[3], stage_factor<2, TW>(t, u, LOGR - 2, 3));
        dft4_dif<TW>(v[0], v[1], v[2], v[3], dk.w4());
        const int rev[4] = {0, 2, 1, 3};
#pragma unroll
        for (int j = 0; j < 4; j++) sm_st(x, u + S * j, fe_canon<FrCfg>(v[rev[j]]));
    }
    __syncthreads();
}

// final radix-2 sub-stage (four items per thread, two at a time), P_s = R / 2
template <int LOGR, class TW>
__device__ __forceinline__ void stage2_last(Fr* x, int lt, const StageTw& t) {
    constexpr int R = 1 << LOGR;
    constexpr int S = R / 2;
    constexpr int TH = R / 8;
    // each thread reads and rewrites only its own slots u and u + S
#pragma unroll 1
    for (int k = 0; k < 4; k += 2) {
        const uint32_t u0 = lt + k * TH, u1 = u0 + TH;
        Fr a0 = sm_ld(x, u0), b0 = sm_ld(x, u0 + S), a1 = sm_ld(x, u1), b1 = sm_ld(x, u1 + S);
        const Fr2 m = TW::mul2(b0, stage_factor<1, TW>(t, u0, LOGR - 1, 1), b1,
                               stage_factor<1, TW>(t, u1, LOGR - 1, 1));
        b0 = m.a;
        b1 = m.b;
        dft2(a0, b0);
        dft2(a1, b1);
        sm_st(x, u0, fe_canon<FrCfg>(a0));
        sm_st(x, u0 + S, fe_canon<FrCfg>(b0));
        sm_st(x, u1, fe_canon<FrCfg>(a1));
        sm_st(x, u1 + S, fe_canon<FrCfg>(b1));
    }
    __syncthreads();
}

// the sub-stages after the first of a DFT of size 2^LOGR in shared memory
template <int LOGR, class TW>
__device__ __forceinline__ void dft_tail(Fr* x, int lt, const StageTw& t, const DftK<TW>& dk) {
    constexpr int NS8 = LOGR / 3;
    constexpr int REM = LOGR % 3;
#pragma unroll 1
    for (int s = 1; s < NS8; s++) {
        Fr v[8];
        stage8_load<LOGR, TW>(v, x, lt);
        stage8_twiddle<TW>(v, t, (uint32_t)lt & ((1u << (3 * s)) - 1), 3 * s);
        stage8_finish<TW>(x, lt, 3 * s, s == NS8 - 1 && REM == 0, v, dk);
    }
    if (REM == 2) stage4_last<LOGR, TW>(x, lt, t, dk);
    if (REM == 1) stage2_last<LOGR, TW>(x, lt, t);
}

#ifndef ZK_PASS10_MIN_BLOCKS
#define ZK_PASS10_MIN_BLOCKS 4
#endif

// resident CTAs per SM the register budget of a pass kernel is sized for:
// 16 warps per SM (128 registers a thread) for most shapes
__host__ __device__ constexpr int pass_min_blocks(int logr, int g) {
    return ((g << logr) / 8) >= 512 ? 1
           : (logr == 10 && g == 1) ? ZK_PASS10_MIN_BLOCKS
           : ((g << logr) / 8 >= 32 ? 512 / ((g << logr) / 8) : 16);
}

template <int LOGR, int G, class TW>
__global__ void __launch_bounds__((G << LOGR) / 8, pass_min_blocks(LOGR, G))
ntt_pass_kernel(NttPassArgs a) {
    constexpr int R = 1 << LOGR;
    constexpr int TR = R / 8;  // threads per DFT
    constexpr int T = G * TR;
    extern __shared__ uint4 smem_u4[];
    Fr* sm = reinterpret_cast<Fr*>(smem_u4);
    const int tid = threadIdx.x;
    const int log_items = a.log_n - LOGR;
    // Blocks run column-fastest: the CTAs of one item across the batch's
    // columns are resident together, so the twiddle and twist values they
    // share are read from DRAM once and from L2 by the other columns (in grid
    // order every column would stream both tables again, 3.5x the pass's
    // algorithmic reads at 8 columns of 2^22).
    const uint64_t lin = (uint64_t)blockIdx.y * gridDim.x + blockIdx.x;
    const uint32_t bx = (uint32_t)(lin / gridDim.y), by = (uint32_t)(lin % gridDim.y);
    const uint32_t q0 = bx * G;
    const Fr* src = a.src + by * a.src_ys + blockIdx.z * a.src_zs;
    Fr* dst = a.dst + by * a.dst_ys + blockIdx.z * a.dst_zs;

    // factors of the first sub-stage's eight inputs, one set an item, where a
    // scale multiplies all eight (times the item's twiddles)
    __shared__ Fr kst[G * 8 * TW::EW];
    __shared__ DftK<TW> dk;
    const bool kst_used = a.scale && !a.in_mul;
    typename DftK<TW>::Raw dk_raw;
    if (T >= 3) dk_raw = DftK<TW>::fetch(tid, a.tw, a.log_n);
    // coalesced load: chunk c -> (i, g, h); global x[q0 + g + (i << log_items)]
    for (int c = tid; c < G * R * 2; c += T) {
        const int h = c & 1, e = c >> 1;
        const int g = e % G, i = e / G;
        const size_t gi = (size_t)(q0 + g) + ((size_t)i << log_items);
        *sm_slot(sm + g * R, i, h) = reinterpret_cast<const uint4*>(src + gi)[h];
    }
    if (T >= 3)
        dk.put(tid, dk_raw);
    else
        dk.init(a.tw, a.log_n);
    if (kst_used) {
        for (int k = tid; k < G * 8; k += T) {
            const uint32_t qk = q0 + k / 8, i = k % 8;
            typename TW::K f = TW::ld(a.scale, 0);
            const uint32_t J = qk & ((1u << a.log_p) - 1);
            if (i * J) f = TW::prod(TW::ld(a.tw, (size_t)(i * J) << (a.log_n - a.log_p - 3)), f);
            TW::put(kst + k * TW::EW, f);
        }
    }
    __syncthreads();

    const int g = tid / TR, lt = tid % TR;
    Fr* x = sm + g * R;
    const uint32_t q = q0 + g;
    const Fr* in_mul = a.in_mul ? TW::off(a.in_mul, blockIdx.z * a.in_mul_zs) : nullptr;
    StageTw st;
    st.tw = a.tw;
    st.ctab = nullptr;
    st.log_n = a.log_n;
    st.log_p = a.log_p;
    st.J = q & ((1u << a.log_p) - 1);

    Fr v[8];
    stage8_load<LOGR, TW>(v, x, lt);
    if (kst_used) {
        stage8_scale<TW>(v, kst + g * 8 * TW::EW);
    } else if (in_mul) {
        // any factors, one an element (the first pass has no twiddles here)
        const size_t m0 = (size_t)q + ((size_t)lt << log_items), ms = (size_t)TR << log_items;
        if constexpr (TW::EW == 2) {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = TW::mul(v[i], TW::ld(in_mul, m0 + i * ms));
        } else {
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                const Fr2 m = TW::mul2(v[i], TW::ld(in_mul, m0 + i * ms), v[i + 1],
                                       TW::ld(in_mul, m0 + (i + 1) * ms));
                v[i] = m.a;
                v[i + 1] = m.b;
            }
        }
        if (a.scale) {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = TW::mul(v[i], TW::ld(a.scale, 0));
        }
    } else {
        stage8_twiddle<TW>(v, st, 0, 0);
    }
    stage8_finish<TW>(x, lt, 0, LOGR == 3, v, dk);
    dft_tail<LOGR, TW>(x, lt, st, dk);

    // coalesced store: dst[(J + P*j + P*R*Q) << out_shift + z*out_off_z]
    const uint32_t pm = (1u << a.log_p) - 1;
    const size_t zoff = (size_t)blockIdx.z * a.out_off_z;
    for (int c = tid; c < G * R * 2; c += T) {
        const int h = c & 1, e = c >> 1;
        int gg, j;
        if (a.log_p == 0) {
            gg = e >> LOGR;
            j = e & (R - 1);
        } else {
            gg = e % G;
            j = e / G;
        }
        const uint32_t qq = q0 + gg;
        const size_t pos = (size_t)(qq & pm) + ((size_t)j << a.log_p) + ((size_t)(qq >> a.log_p) << (a.log_p + LOGR));
        const size_t o = (pos << a.out_shift) + zoff;
        reinterpret_cast<uint4*>(dst + o)[h] = *sm_slot(sm + gg * R, j, h);
    }
}

// Fused extended-domain stage.  For one column and work item q it runs
//   (1) the last pass of the inverse transform: radix R = 2^LOGR, P = n/R,
//       input tmp[q + (n/R) i], output the coefficients c[q + (n/R) j] * n^-1,
//       written to coeff;
//   (2) for each coset z, the first pass of that coset's forward transform in
//       the reversed radix order (radix R first, P = 1), whose item q reads
//       exactly the same coefficients c[q + (n/R) i], to be multiplied by
//       t_z^(q + (n/R) i): the first sub-stage's eight inputs take
//       t_z^q (t_z^(n/8))^i (W_z[q R] S_z[(R/8) i], eight factors a coset made
//       at the start), the later sub-stages ctab's factors; then written to
//       sub[z n + y + R q].
// The coefficients stay on the CTA's tile for the first coset; later cosets
// re-read them from L2.
// resident CTAs per SM the register budget is sized for: one tile a CTA (the
// coefficients re-read from L2 for each coset) allows 7 of 2^9, 4 of 2^10 and,
// at 128 registers a thread, 2 of 2^11
#ifndef ZK_FUSED11_MIN_BLOCKS
#define ZK_FUSED11_MIN_BLOCKS 2
#endif
__host__ __device__ constexpr int fused_min_blocks(int logr) {
    return logr <= 9 ? 7 : logr == 10 ? 4 : ZK_FUSED11_MIN_BLOCKS;
}

static constexpr int FUSED_MAX_E = 16;

template <int LOGR, class TW>
__global__ void __launch_bounds__((1 << LOGR) / 8, fused_min_blocks(LOGR))
ntt_fused_extend_kernel(FusedExtendArgs a) {
    constexpr int R = 1 << LOGR;
    constexpr int T = R / 8;
    extern __shared__ uint4 smem_u4[];
    Fr* A = reinterpret_cast<Fr*>(smem_u4);
    __shared__ Fr kst[8 * (1 + FUSED_MAX_E) * TW::EW];  // the inverse pass's factors, then each coset's
    __shared__ DftK<TW> dki, dkf;
    const int tid = threadIdx.x;
    const int log_items = a.log_n - LOGR;
    // column-fastest block order, as in ntt_pass_kernel: the per-coset tables
    // an item reads are shared by every column of the launch
    const uint64_t lin = (uint64_t)blockIdx.y * gridDim.x + blockIdx.x;
    const uint32_t q = (uint32_t)(lin / gridDim.y), col = (uint32_t)(lin % gridDim.y);
    const size_t n = (size_t)1 << a.log_n;
    const Fr* src = a.src + col * a.src_ys;
    Fr* coeff = a.coeff + col * a.coeff_ys;
    Fr* sub = a.sub + col * a.sub_ys;

    for (int c = tid; c < R * 2; c += T) {
        const int h = c & 1, i = c >> 1;
        *sm_slot(A, i, h) = reinterpret_cast<const uint4*>(src + q + ((size_t)i << log_items))[h];
    }
    dki.init(a.tw_inv, a.log_n);
    dkf.init(a.tw, a.log_n);
    for (int k = tid; k < 8 * (1 + a.E); k += T) {
        const uint32_t i = k % 8;
        typename TW::K f;
        if (k < 8) {
            f = TW::ld(a.n_inv, 0);
            if (i * q) f = TW::prod(TW::ld(a.tw_inv, (size_t)(i * q) << (LOGR - 3)), f);
        } else {
            const size_t z = k / 8 - 1;
            f = TW::ld(a.wtab, z * n + (size_t)q * R);
            if (i) f = TW::prod(TW::ld(a.stab, z * R + (size_t)(R / 8) * i), f);
        }
        TW::put(kst + k * TW::EW, f);
    }
    __syncthreads();
    StageTw st;
    st.tw = a.tw_inv;
    st.ctab = nullptr;
    st.log_n = a.log_n;
    st.log_p = log_items;
    st.J = q;
    Fr v[8];
    stage8_load<LOGR, TW>(v, A, tid);
    stage8_scale<TW>(v, kst);
    stage8_finish<TW>(A, tid, 0, false, v, dki);
    dft_tail<LOGR, TW>(A, tid, st, dki);
    for (int c = tid; c < R * 2; c += T) {
        const int h = c & 1, j = c >> 1;
        reinterpret_cast<uint4*>(coeff + q + ((size_t)j << log_items))[h] = *sm_slot(A, j, h);
    }
    st.tw = a.tw;
    st.log_p = 0;
    st.J = 0;
    for (int z = 0; z < a.E; z++) {
        // coset 0 reads the tile; later cosets the coefficients this CTA wrote
        // (the barrier below orders the writes of its other threads)
        if (z == 0) {
            stage8_load<LOGR, TW>(v, A, tid);
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++)
                v[i] = ld_elem<FrCfg>(coeff + q + ((size_t)(tid + (R / 8) * i) << log_items));
        }
        st.ctab = TW::off(a.ctab, (size_t)z * 2 * R);
        stage8_scale<TW>(v, kst + 8 * (1 + z) * TW::EW);
        stage8_finish<TW>(A, tid, 0, false, v, dkf);
        dft_tail<LOGR, TW>(A, tid, st, dkf);
        Fr* out = sub + (size_t)z * n + (size_t)q * R;
        for (int c = tid; c < R * 2; c += T) {
            const int h = c & 1, y = c >> 1;
            reinterpret_cast<uint4*>(out + y)[h] = *sm_slot(A, y, h);
        }
        __syncthreads();
    }
}

template <int LOGR, class TW>
static cudaError_t launch_fused(const FusedExtendArgs& a, unsigned ncols, cudaStream_t s) {
    constexpr int R = 1 << LOGR;
    const size_t smem = (size_t)R * sizeof(Fr);
    static SmemOptIn opt;
    ZK_CHECK(opt.ensure(ntt_fused_extend_kernel<LOGR, TW>, (int)smem));
    dim3 grid(1u << (a.log_n - LOGR), ncols, 1);
    ntt_fused_extend_kernel<LOGR, TW><<<grid, R / 8, smem, s>>>(a);
    return cudaGetLastError();
}

template <class TW>
static cudaError_t fused_dispatch(const FusedExtendArgs& a, int log_r, unsigned ncols, cudaStream_t s) {
    switch (log_r) {
        case 9: return launch_fused<9, TW>(a, ncols, s);
        case 10: return launch_fused<10, TW>(a, ncols, s);
        case 11: return launch_fused<11, TW>(a, ncols, s);
        default: return cudaErrorInvalidValue;
    }
}

// Factors of the sub-stages after the first in the first pass (radix R = 2^log_r)
// of a coset transform X[j] = sum_k x_k s^k w_n^(jk).  In that pass item q's
// DFT runs over x_(q + (n/R) i) s^((n/R) i) (s^q goes into its first
// sub-stage), so a sub-stage of radix r after P_s multiplies input i of local
// item Jl by s^(i n/(P_s r)) w_(P_s r)^(i Jl): the same factors for every q and
// column, at entry r (P_s + Jl) + i, 2 R entries a coset.  pw holds the R powers
// of s^(n/R), so s^k is its entry k >> pw_shift, pw_shift = log2(n/R).
// Made once per call into a buffer the first pass does not write.
template <class TW>
__global__ void ntt_coset_table_kernel(Fr* ctab, const Fr* pw, size_t pw_zs, int pw_shift, const Fr* tw, int log_n,
                                       int log_r) {
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 2u << log_r) return;
    // the sub-stages' P_s are 8, 64, ... and the last one's radix is 8, 4 or 2
    int log_ps = 3, lr = 3;
    for (; log_ps < log_r; log_ps += 3) {
        lr = log_r - log_ps < 3 ? log_r - log_ps : 3;
        if (e >> lr >= 1u << log_ps && e >> lr < 2u << log_ps) break;
    }
    if (log_ps >= log_r) return;  // a gap between two sub-stages' entries
    const uint32_t Jl = (e >> lr) - (1u << log_ps), i = e & ((1u << lr) - 1);
    const size_t k = (size_t)i << (log_n - log_ps - lr);
    typename TW::K f = TW::ld(TW::off(pw, blockIdx.y * pw_zs), k >> pw_shift);
    if (i * Jl) f = TW::prod(TW::ld(tw, (size_t)(i * Jl) << (log_n - log_ps - lr)), f);
    TW::put(ctab + ((size_t)blockIdx.y * (2u << log_r) + e) * TW::EW, f);
}

cudaError_t ntt_coset_table(Fr* ctab, const Fr* pw, size_t pw_zs, int pw_shift, const Fr* tw, int log_n, int log_r,
                            int cosets, int pairs, cudaStream_t s) {
    const dim3 grid(((2u << log_r) + 127) / 128, cosets);
    if (pairs)
        ntt_coset_table_kernel<TwS><<<grid, 128, 0, s>>>(ctab, pw, pw_zs, pw_shift, tw, log_n, log_r);
    else
        ntt_coset_table_kernel<TwM><<<grid, 128, 0, s>>>(ctab, pw, pw_zs, pw_shift, tw, log_n, log_r);
    return cudaGetLastError();
}

cudaError_t ntt_fused_extend(const FusedExtendArgs& a, int log_r, unsigned ncols, cudaStream_t s) {
    if (a.E > FUSED_MAX_E) return cudaErrorInvalidValue;
    return a.pairs ? fused_dispatch<TwS>(a, log_r, ncols, s) : fused_dispatch<TwM>(a, log_r, ncols, s);
}

// Tables of the fused stage for radix R = 2^log_r: wtab[z n + q R + y] =
// w^(q y) t_z^q (q < n/R, y < R) and stab[z R + i] = (t_z^(n/R))^i, with
// t_z = shift * w_ext^z and w^k read from the natural table tw.
template <bool PAIRS>
__global__ void fused_tables_kernel(Fr* wtab, Fr* stab, const Fr* tw, const Fr* shift, const Fr* w_ext, int log_n,
                                    int log_r) {
    const uint32_t z = blockIdx.y;
    const uint32_t R = 1u << log_r;
    const uint32_t items = 1u << (log_n - log_r);
    const size_t n = (size_t)1 << log_n;
    const Fr tz = nt_mul(ld_elem<FrCfg>(shift), fe_pow_u32<FrCfg>(ld_elem<FrCfg>(w_ext), z));
    for (uint32_t q = blockIdx.x; q < items; q += gridDim.x) {
        const Fr tq = fe_pow_u32<FrCfg>(tz, q);
        for (uint32_t y = threadIdx.x; y < R; y += blockDim.x) {
            const Fr w = ld_elem<FrCfg>(tw + (size_t)q * y);
            st_factor<PAIRS>(wtab, (size_t)z * n + (size_t)q * R + y, y == 0 ? tq : nt_mul(w, tq));
        }
    }
    if (blockIdx.x == 0) {
        const Fr s = fe_pow_u32<FrCfg>(tz, items);
        for (uint32_t i = threadIdx.x; i < R; i += blockDim.x)
            st_factor<PAIRS>(stab, (size_t)z * R + i, fe_pow_u32<FrCfg>(s, i));
    }
}

cudaError_t ntt_fused_tables(Fr* wtab, Fr* stab, const Fr* tw, const Fr* shift, const Fr* w_ext, int log_n, int log_r,
                             int ext_bits, cudaStream_t s, bool pairs) {
    const uint32_t items = 1u << (log_n - log_r);
    dim3 grid(items < 4096 ? items : 4096, 1u << ext_bits);
    if (pairs)
        fused_tables_kernel<true><<<grid, 256, 0, s>>>(wtab, stab, tw, shift, w_ext, log_n, log_r);
    else
        fused_tables_kernel<false><<<grid, 256, 0, s>>>(wtab, stab, tw, shift, w_ext, log_n, log_r);
    return cudaGetLastError();
}

// out[i] = (w, w') for the Montgomery-form factors in[i], i < n
__global__ void shoup_pairs_kernel(Fr* out, const Fr* in, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        st_factor<true>(out, i, ld_elem<FrCfg>(in + i));
}

cudaError_t shoup_pairs(Fr* out, const Fr* in, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const size_t blocks = (n + 255) / 256;
    shoup_pairs_kernel<<<(unsigned)(blocks < 148 * 32 ? blocks : 148 * 32), 256, 0, s>>>(out, in, n);
    return cudaGetLastError();
}

// ------------------------------------------------------------ short passes
// A pass for transforms too small to fill the SMs (up to NTT_SHORT elements in
// all), where the time is one thread's chain of products: radix-2 sub-stages,
// two elements a thread, so a level costs one product where the radix-8 form's
// threads take eleven for three levels, on four times the threads.  A thread's
// twiddles of every level are read at the start and the products are inline
// (13.8 us through the out-of-line product).  One column of 2^13: 12.3 us
// against 45.8 in radix-8 sub-stages.  The line
// is where the columns' n / 2 threads come to 1024 warps, two for each of the
// SMs' four schedulers.
static constexpr uint32_t NTT_SHORT = 1u << 16;

template <int LOGR>
__host__ __device__ constexpr int short_group() {
    return LOGR >= 7 ? 1 : 64 >> (LOGR - 1);  // 64 threads a CTA
}

template <int LOGR>
__global__ void __launch_bounds__((short_group<LOGR>() << LOGR) / 2) ntt_short_pass_kernel(NttPassArgs a) {
    constexpr int R = 1 << LOGR, H = R / 2, G = short_group<LOGR>();
    __shared__ Fr tile[2][G * R];
    const int g = threadIdx.x / H, u = threadIdx.x % H;
    const uint32_t q = blockIdx.x * G + g;
    const int log_items = a.log_n - LOGR;
    const uint32_t J = q & ((1u << a.log_p) - 1);
    const Fr* src = a.src + blockIdx.y * a.src_ys + blockIdx.z * a.src_zs;
    Fr* dst = a.dst + blockIdx.y * a.dst_ys + blockIdx.z * a.dst_zs;
    const size_t i0 = (size_t)q + ((size_t)u << log_items), i1 = i0 + ((size_t)H << log_items);
    Fr x = ld_elem<FrCfg>(src + i0), y = ld_elem<FrCfg>(src + i1);
    Fr w[LOGR];
#pragma unroll
    for (int s = 0; s < LOGR; s++) {
        const uint32_t Jl = (uint32_t)u & ((1u << s) - 1);
        w[s] = ldg_elem<FrCfg>(a.tw + ((size_t)(J + (Jl << a.log_p)) << (a.log_n - a.log_p - s - 1)));
    }
    if (a.in_mul) {
        const Fr* m = a.in_mul + blockIdx.z * a.in_mul_zs;
        x = fe_mul_lazy<FrCfg>(x, ldg_elem<FrCfg>(m + i0));
        y = fe_mul_lazy<FrCfg>(y, ldg_elem<FrCfg>(m + i1));
    }
    if (a.scale) {
        const Fr sc = ldg_elem<FrCfg>(a.scale);
        x = fe_mul_lazy<FrCfg>(x, sc);
        w[0] = fe_mul_lazy<FrCfg>(w[0], sc);
    }
#pragma unroll
    for (int s = 0; s < LOGR; s++) {
        const uint32_t Jl = (uint32_t)u & ((1u << s) - 1), ilo = (uint32_t)u >> s;
        // (the first sub-stage of an unscaled first pass has factor one)
        if (s > 0 || J || a.scale) y = fe_mul_lazy<FrCfg>(y, w[s]);
        dft2(x, y);
        if (s + 1 < LOGR) {
            Fr* t = tile[s & 1] + g * R;
            const uint32_t pos = Jl + (ilo << (s + 1));
            sm_st(t, pos, x);
            sm_st(t, pos + (1u << s), y);
            __syncthreads();
            x = sm_ld(t, u);
            y = sm_ld(t, u + H);
        }
    }
    const size_t pos = (size_t)J + ((size_t)u << a.log_p) + ((size_t)(q >> a.log_p) << (a.log_p + LOGR));
    const size_t zoff = (size_t)blockIdx.z * a.out_off_z;
    st_elem<FrCfg>(dst + ((pos << a.out_shift) + zoff), fe_canon<FrCfg>(x));
    st_elem<FrCfg>(dst + (((pos + ((size_t)H << a.log_p)) << a.out_shift) + zoff), fe_canon<FrCfg>(y));
}

template <int LOGR>
static cudaError_t launch_short(const NttPassArgs& a, unsigned ny, unsigned nz, cudaStream_t s) {
    constexpr int G = short_group<LOGR>();
    ntt_short_pass_kernel<LOGR><<<dim3((1u << (a.log_n - LOGR)) / G, ny, nz), (G << LOGR) / 2, 0, s>>>(a);
    return cudaGetLastError();
}

bool ntt_is_short(int log_n, uint64_t transforms) { return (transforms << log_n) <= NTT_SHORT; }

// tiny transforms (n <= 4): direct O(n^2) evaluation by one thread per column
__global__ void ntt_tiny_kernel(NttPassArgs a) {
    const int n = 1 << a.log_n;
    const Fr* src = a.src + blockIdx.y * a.src_ys;
    Fr* dst = a.dst + blockIdx.y * a.dst_ys;
    if (threadIdx.x != 0) return;
    Fr x[4], y[4];
    for (int i = 0; i < n; i++) {
        x[i] = ld_elem<FrCfg>(src + i);
        if (a.in_mul) x[i] = nt_mul(x[i], ld_elem<FrCfg>(a.in_mul + i));
    }
    for (int j = 0; j < n; j++) {
        Fr acc = fe_zero<FrCfg>();
        for (int i = 0; i < n; i++) {
            Fr t = x[i];
            int e = (i * j) & (n - 1);
            if (e) t = nt_mul(t, ld_elem<FrCfg>(a.tw + e));
            acc = fe_add<FrCfg>(acc, t);
        }
        if (a.scale) acc = nt_mul(acc, ld_elem<FrCfg>(a.scale));
        y[j] = acc;
    }
    for (int j = 0; j < n; j++) st_elem<FrCfg>(dst + ((size_t)j << a.out_shift), y[j]);
}

// ---------------------------------------------------------------- launchers

template <int LOGR, int G, class TW>
static cudaError_t launch_pass(const NttPassArgs& a, unsigned ny, unsigned nz, cudaStream_t s) {
    constexpr int R = 1 << LOGR;
    constexpr int T = (G * R) / 8;
    const size_t smem = (size_t)G * R * sizeof(Fr);
    static SmemOptIn opt;
    ZK_CHECK(opt.ensure(ntt_pass_kernel<LOGR, G, TW>, (int)smem));
    const unsigned items = 1u << (a.log_n - LOGR);
    dim3 grid(items / G, ny, nz);
    ntt_pass_kernel<LOGR, G, TW><<<grid, T, smem, s>>>(a);
    return cudaGetLastError();
}

// Items per CTA: about 1024 elements, so that a CTA's rows are read in runs of
// several elements; fewer where that leaves the SMs without a CTA each (one
// column of 2^13: 8 CTAs), down to one warp a CTA, since a warp's chain of
// products takes the same time alone or beside three others.
static int pass_group(int log_r, int log_n, unsigned cols) {
    int g = 1;
    if (log_r <= 9) g = 1 << (10 - log_r);
    if (g > 16) g = 16;
    const int items = 1 << (log_n - log_r);
    if (g > items) g = items;
    while (g > 1 && (g << log_r) > 256 && (uint64_t)(items / g) * cols < 148) g /= 2;
    return g;
}

template <class TW>
static cudaError_t pass_dispatch(const NttPassArgs& a, int log_r, unsigned ny, unsigned nz, cudaStream_t s) {
    const int g = pass_group(log_r, a.log_n, ny * nz);
#define ZK_PASS(LR, GG) \
    if (log_r == LR && g == GG) return launch_pass<LR, GG, TW>(a, ny, nz, s);
    ZK_PASS(3, 1) ZK_PASS(4, 1) ZK_PASS(5, 1) ZK_PASS(6, 1) ZK_PASS(7, 1) ZK_PASS(8, 1)
    ZK_PASS(9, 1) ZK_PASS(10, 1) ZK_PASS(11, 1) ZK_PASS(12, 1)
    ZK_PASS(6, 2) ZK_PASS(6, 4) ZK_PASS(6, 8) ZK_PASS(6, 16)
    ZK_PASS(7, 2) ZK_PASS(7, 4) ZK_PASS(7, 8)
    ZK_PASS(8, 2) ZK_PASS(8, 4)
    ZK_PASS(9, 2)
#undef ZK_PASS
    return cudaErrorInvalidValue;
}

cudaError_t ntt_pass(const NttPassArgs& a, int log_r, unsigned ny, unsigned nz, cudaStream_t s) {
    if (a.log_n <= 2) {
        if (a.pairs) return cudaErrorInvalidValue;  // the direct kernel reads Montgomery tables
        ntt_tiny_kernel<<<dim3(1, ny, nz), 32, 0, s>>>(a);
        return cudaGetLastError();
    }
    if (!a.pairs && ntt_is_short(a.log_n, (uint64_t)ny * nz)) {
        // (where the items are a CTA's at least: two passes)
        if (log_r == 5 && a.log_n >= 5 + 2) return launch_short<5>(a, ny, nz, s);
        if (log_r == 6 && a.log_n >= 6 + 1) return launch_short<6>(a, ny, nz, s);
        if (log_r == 7) return launch_short<7>(a, ny, nz, s);
        if (log_r == 8) return launch_short<8>(a, ny, nz, s);
        if (log_r == 9) return launch_short<9>(a, ny, nz, s);
    }
    return a.pairs ? pass_dispatch<TwS>(a, log_r, ny, nz, s) : pass_dispatch<TwM>(a, log_r, ny, nz, s);
}

// split log_n into pass radices (at most ZK_NTT_MAX_PASS_BITS bits per pass,
// as even as possible).  11: 2^24 runs as three passes of 2^8 (4.25 ms on
// B200) rather than two of 2^12 (4.78 ms; one 512-thread CTA of 128 KB per
// SM); 10 would slow 2^21 and 2^22.
#ifndef ZK_NTT_MAX_PASS_BITS
#define ZK_NTT_MAX_PASS_BITS 11
#endif
// The splits the radix autotuner (zkp_ntt_batch_plan over every split into
// 2-3 passes of 2^6..2^12, one column) measured fastest on B200 for 2^13..2^25,
// with passes whose twiddles came after the DFT; other sizes use the even split
// below, columns of up to NTT_SHORT elements in all two even passes (ntt_run).
static const int8_t TUNED_SPLIT[13][3] = {{7, 6, 0},  {6, 8, 0},  {6, 9, 0},   {8, 8, 0},  {8, 9, 0},
                                          {9, 9, 0},  {11, 8, 0}, {10, 10, 0}, {11, 10, 0}, {11, 11, 0},
                                          {11, 6, 6}, {9, 9, 6},  {9, 10, 6}};

int ntt_plan(int log_n, int radices[4]) {
    if (log_n <= 12) {
        radices[0] = log_n;
        return 1;
    }
    if (log_n <= 25) {
        const int8_t* t = TUNED_SPLIT[log_n - 13];
        const int np = t[2] ? 3 : 2;
        for (int i = 0; i < np; i++) radices[i] = t[i];
        return np;
    }
    int np = (log_n + ZK_NTT_MAX_PASS_BITS - 1) / ZK_NTT_MAX_PASS_BITS;
    if (np < 2) np = 2;
    for (int i = 0; i < np; i++) radices[i] = log_n / np + (i < log_n % np ? 1 : 0);
    return np;
}

cudaError_t ntt_run(Fr* buf, Fr* tmp, const Fr* tw, const Fr* scale, int log_n, unsigned ncols,
                    size_t col_stride, bool* result_in_tmp, cudaStream_t s) {
    int rad[4];
    const int np = ntt_plan(log_n, rad);
    if (np == 2 && ntt_is_short(log_n, ncols)) {
        // two even passes on as many SMs as the columns fill (the result is in buf
        // either way).  Transforms of one pass keep it: tmp is not theirs to write.
        rad[0] = (log_n + 1) / 2;
        rad[1] = log_n / 2;
        return ntt_run_plan(buf, tmp, tw, scale, log_n, ncols, col_stride, rad, 2, result_in_tmp, s);
    }
    return ntt_run_plan(buf, tmp, tw, scale, log_n, ncols, col_stride, rad, np, result_in_tmp, s);
}

cudaError_t ntt_run_plan(Fr* buf, Fr* tmp, const Fr* tw, const Fr* scale, int log_n, unsigned ncols,
                         size_t col_stride, const int* rad, int np, bool* result_in_tmp, cudaStream_t s) {
    int log_p = 0;
    for (int p = 0; p < np; p++) {
        // one pass runs in place; otherwise ping-pong buf -> tmp -> buf ...
        Fr* src = (np == 1 || p % 2 == 0) ? buf : tmp;
        Fr* dst = (np == 1) ? buf : (p % 2 == 0 ? tmp : buf);
        NttPassArgs a = {};
        a.src = src;
        a.dst = dst;
        a.tw = tw;
        a.log_n = log_n;
        a.log_p = log_p;
        a.scale = (p == np - 1) ? scale : nullptr;
        a.src_ys = col_stride;
        a.dst_ys = col_stride;
        ZK_CHECK(ntt_pass(a, rad[p], ncols, 1, s));
        log_p += rad[p];
    }
    *result_in_tmp = (np > 1) && (np % 2 == 1);
    return cudaSuccess;
}

// ---------------------------------------------------------------- tables

// Geometric sequences out[i] = base * w^i for i0 <= i < n (base null: 1) in
// two launches, one product per element instead of a power per thread:
//   coarse  out[k C] for every k: a thread takes GEO_C2 consecutive k, starts
//           from one power and steps by w^C;
//   fine    the run out[k C + 1 .. k C + C - 1] from out[k C] by steps of w.
// Each run is C dependent products on one thread, and the thread count stays
// n / C.
static constexpr uint32_t GEO_C = 64;
static constexpr uint32_t GEO_C2 = 64;

__device__ __forceinline__ Fr geo_base(const Fr* base) { return base ? ld_elem<FrCfg>(base) : fe_one<FrCfg>(); }

__global__ void geo_coarse_kernel(Fr* out, const Fr* base, const Fr* w, uint32_t n, uint32_t i0) {
    const uint64_t k0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * GEO_C2;
    if (k0 * GEO_C >= n) return;
    const Fr r = fe_pow_u32<FrCfg>(ld_elem<FrCfg>(w), GEO_C);
    Fr cur = nt_mul(geo_base(base), fe_pow_u32<FrCfg>(r, (uint32_t)k0));
    for (uint64_t k = k0; k < k0 + GEO_C2 && k * GEO_C < n; k++) {
        if (k * GEO_C >= i0) st_elem<FrCfg>(out + k * GEO_C, cur);
        cur = nt_mul(cur, r);
    }
}

__global__ void geo_fine_kernel(Fr* out, const Fr* base, const Fr* w, uint32_t n, uint32_t i0) {
    const uint64_t s = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * GEO_C;
    if (s >= n) return;
    const Fr ww = ld_elem<FrCfg>(w);
    // a run start below i0 was not written by the coarse pass
    Fr cur = s >= i0 ? ld_elem<FrCfg>(out + s) : nt_mul(geo_base(base), fe_pow_u32<FrCfg>(ww, (uint32_t)s));
    for (uint64_t i = s + 1; i < s + GEO_C && i < n; i++) {
        cur = nt_mul(cur, ww);
        if (i >= i0) st_elem<FrCfg>(out + i, cur);
    }
}

static cudaError_t geometric_from(Fr* out, const Fr* base, const Fr* w, uint32_t n, uint32_t i0, cudaStream_t s) {
    if (n <= i0) return cudaSuccess;
    const uint64_t runs = (n + GEO_C - 1) / GEO_C;
    const uint64_t coarse = (runs + GEO_C2 - 1) / GEO_C2;
    geo_coarse_kernel<<<(unsigned)((coarse + 127) / 128), 128, 0, s>>>(out, base, w, n, i0);
    ZK_CHECK(cudaGetLastError());
    geo_fine_kernel<<<(unsigned)((runs + 127) / 128), 128, 0, s>>>(out, base, w, n, i0);
    return cudaGetLastError();
}

// buf[i] = w^i for 2 <= i < n, with w = buf[1] (entries 0 and 1 written by the
// host and left as they are)
cudaError_t expand_powers(Fr* buf, uint32_t n, cudaStream_t s) { return geometric_from(buf, nullptr, buf + 1, n, 2, s); }

// out[i] = base * w^i for i < n, w and base given by value in device memory
cudaError_t geometric(Fr* out, const Fr* base, const Fr* w, uint32_t n, cudaStream_t s) {
    return geometric_from(out, base, w, n, 0, s);
}

}  // namespace zk
