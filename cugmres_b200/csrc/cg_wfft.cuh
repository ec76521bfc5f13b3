// Warp-level FFTs of the circulant embedding, for kernels that keep whole lines
// within a warp (cg_small.cu).
//
// An embedding of side L = 2 NP is never transformed as a length-L line.  A line
// whose upper half is zero has the length-L spectrum
//
//   X[2 m + p] = FFT_NP( x[n] w_L^{p n} )[m],   p = 0, 1,
//
// and a line of which only the first NP values are wanted has the inverse
//
//   x[n] = IFFT_NP( X[2 m] )[n] + w_L^{-n} IFFT_NP( X[2 m + 1] )[n],
//
// so both directions are two independent transforms of length NP (one per
// parity p) and neither the padding nor the cropped half is ever touched.
//
// NP = 64 = R R with R = 8: eight lanes run a transform, four transforms a warp, eight
// values per lane; one radix-8 stage, one exchange through the warp's own piece of
// shared memory, one radix-8 stage, synchronising the warp's lanes only.  That is the
// shortest chain there is for short lines, where cg_fft.cuh's block-wide stages wait
// at two barriers each.
//
// Index maps.  Lane t of a transform holds in register i the element t + R i, on
// entry and on exit, forward and inverse.
//   stage 1: butterfly t over elements t + R r, r < R, gives q < R
//   twiddle: w_NP^{t q}, times w_L^{p t} (forward) or w_L^{p q} (inverse)
//   exchange: element (q, j) at q (R + 1) + j   (odd pitch: no bank conflicts)
//   stage 2: butterfly q = t over j < R, gives s; element q + R s.
// The parity factor w_L^{p n} splits into w_L^{p t}, which joins the stage
// twiddle, and w_{2 R}^{p r}, a compile-time constant per register (forward:
// on the inputs, n = t + R r; inverse: on the outputs, n = q + R s).
#pragma once

#include "cg_common.cuh"

namespace cg {

// ------------------------------------------------------------ constants
// cos(2 pi k / 16) for any integer k (exact decimal expansions).
__host__ __device__ constexpr double cos16(int k) {
    constexpr double tab[5] = {1.000000000000000000000, 0.923879532511286756128, 0.707106781186547524400,
                               0.382683432365089771728, 0.0};
    k &= 15;
    if (k > 8) k = 16 - k;
    return k <= 4 ? tab[k] : -tab[8 - k];
}
__host__ __device__ constexpr double sin16(int k) { return cos16(k - 4); }

// a * exp(-/+ 2 pi i K / 16) (forward / inverse), 0 <= K < 8
template <int K, bool INV, typename C> __device__ __forceinline__ C mul_const(C a) {
    typedef typename real_of<C>::type R;
    if constexpr (K == 0) {
        return a;
    } else if constexpr (K == 4) {
        return INV ? mk<C>(-a.y, a.x) : mk<C>(a.y, -a.x);
    } else {
        constexpr R c = (R)cos16(K), s = (R)(INV ? sin16(K) : -sin16(K));
        return mk<C>(fma_r(a.x, c, -a.y * s), fma_r(a.x, s, a.y * c));
    }
}

// (e + w o, e - w o), w = exp(-/+ 2 pi i K / 16), K = 0, 2, 4, 6.  At 2 and 6 cosine and
// sine have one modulus m: w o = m (o.x -+ o.y, o.y +- o.x), six operations.
template <int K, bool INV, typename C> __device__ __forceinline__ void bfly(C e, C o, C &a, C &b) {
    typedef typename real_of<C>::type R;
    static_assert(K >= 0 && K < 8 && K % 2 == 0, "eighths of a turn");
    if constexpr (K % 4 == 0) {
        const C t = mul_const<K, INV>(o);
        a = cadd(e, t);
        b = csub(e, t);
    } else {
        constexpr double c = cos16(K), s = INV ? sin16(K) : -sin16(K);
        constexpr R m = (R)c;
        constexpr bool same = (c > 0) == (s > 0);
        const R tx = same ? o.x - o.y : o.x + o.y, ty = same ? o.y + o.x : o.y - o.x;
        a = mk<C>(fma_r(m, tx, e.x), fma_r(m, ty, e.y));
        b = mk<C>(fma_r(-m, tx, e.x), fma_r(-m, ty, e.y));
    }
}

template <int R, int K, bool INV, typename C> __device__ __forceinline__ void wcombine(const C *e, const C *o, C *v) {
    if constexpr (K < R / 2) {
        bfly<K * (16 / R), INV>(e[K], o[K], v[K], v[K + R / 2]);
        wcombine<R, K + 1, INV>(e, o, v);
    }
}

// In-place natural-order DFT of R <= 8 values in registers, unscaled.
template <int R, bool INV, typename C> __device__ __forceinline__ void wdft(C *v) {
    if constexpr (R > 1) {
        C e[R / 2], o[R / 2];
#pragma unroll
        for (int i = 0; i < R / 2; i++) {
            e[i] = v[2 * i];
            o[i] = v[2 * i + 1];
        }
        wdft<R / 2, INV>(e);
        wdft<R / 2, INV>(o);
        wcombine<R, 0, INV>(e, o, v);
    }
}

// v[i] *= exp(-/+ 2 pi i i / 16) for i = I .. 7
template <int I, bool INV, typename C> __device__ __forceinline__ void wscale(C *v) {
    if constexpr (I < 8) {
        v[I] = mul_const<I, INV>(v[I]);
        wscale<I + 1, INV>(v);
    }
}

// ------------------------------------------------------------ plan
struct WPlan {
    static constexpr int NP = 64, L = 2 * NP, R = 8;
    static constexpr int E = R;           // values per lane
    static constexpr int LPT = R;         // lanes per transform
    static constexpr int TPW = 32 / LPT;  // transforms per warp
    // exchange region of one transform; the regions of a warp start LPT elements
    // apart modulo 16, so that the 16 lanes of an 8-byte phase (8 lanes of a 16-byte
    // one) stay on distinct banks
    static constexpr int REG = R * (R + 1);
    static constexpr int WREG = TPW * REG;  // elements of a warp's region
    static_assert(R * R == NP && REG % 16 == LPT && WREG >= 32 * E, "two-stage plan");
};

// Twiddle tables of one precision, entries exp(-2 pi i m / L) for the lane index l and
// the register index a of stage 1's outputs: forward [p][a][l], m = l (2 a + p),
// then inverse [p][a][l], m = a (2 l + p).  Consecutive lanes read consecutive entries.
constexpr int WTW_HALF = 2 * WPlan::R * WPlan::R, WTW_ENTRIES = 2 * WTW_HALF;
__host__ __device__ inline int wtw_exponent(int i) {
    constexpr int R = WPlan::R;
    const bool inv = i >= WTW_HALF;
    const int p = i / (R * R) % 2, a = i / R % R, l = i % R;
    return (inv ? a * (2 * l + p) : l * (2 * a + p)) % WPlan::L;
}

// v[a] *= the stage twiddle of lane l and parity p (conjugate for INV)
template <bool INV, typename C>
__device__ __forceinline__ void wtwiddle(C (&v)[WPlan::R], const C *__restrict__ tw, int l, int p) {
    constexpr int R = WPlan::R;
    const C *t = tw + (INV ? WTW_HALF : 0) + p * (R * R) + l;
#pragma unroll
    for (int a = 0; a < R; a++) {
        C w = __ldg(t + a * R);
        if constexpr (INV) w = cconj(w);
        v[a] = cmul(v[a], w);
    }
}

// One length-NP transform of parity p (p is uniform over the warp) in registers as
// above: forward takes x[n] and gives X[2 m + p]; inverse takes X[2 m + p] and gives
// w_L^{-p n} IFFT_NP(...)[n].  sm: the warp's exchange region; t: lane within the
// transform; u: transform within the warp.  The region may be written again after
// __syncwarp().
template <bool INV, typename C>
__device__ __forceinline__ void wfft(C (&reg)[WPlan::E], C *sm, const C *__restrict__ tw, int t, int u, int p) {
    constexpr int R = WPlan::R;
    C *x = sm + u * WPlan::REG;
    if constexpr (!INV) {
        if (p) wscale<1, false>(reg);  // w_{2 R}^r
    }
    wdft<R, INV>(reg);
    wtwiddle<INV>(reg, tw, t, p);  // w_L^{t (2 q + p)}, inverse w_L^{-q (2 t + p)}
#pragma unroll
    for (int q = 0; q < R; q++) x[q * (R + 1) + t] = reg[q];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < R; j++) reg[j] = x[t * (R + 1) + j];
    wdft<R, INV>(reg);
    if constexpr (INV) {
        if (p) wscale<1, true>(reg);  // w_{2 R}^{-s}
    }
}

}  // namespace cg
