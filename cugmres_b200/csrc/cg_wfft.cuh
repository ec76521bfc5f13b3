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
// A warp runs 32 / LPT transforms of length NP, LPT lanes each: E values per lane,
// one radix-R1 stage, one exchange through the warp's own piece of shared memory,
// one radix-R2 stage (NP = R1 R2, E = the larger radix), synchronising its own
// lanes only.  That is the shortest chain there is for short lines, where
// cg_fft.cuh's block-wide stages wait at two barriers each; for L >= 512 in FP64 the
// 16 to 32 values per lane leave too few warps per SM (L = 2048: a product of three
// passes 95.6 us by cg_fft.cuh, 92.5 to 108 by these).
//
// Index maps.  Lane t of a transform holds in register p the element
// t + p LPT, on entry and on exit, forward and inverse ("canonical").
//   stage 1: butterfly j = t + b LPT over elements j + R2 r, r < R1, gives q < R1
//   twiddle: w_NP^{j q}, times w_L^{p j} (forward) or w_L^{p q} (inverse); j = t, since LPT = R2
//   exchange: element (q, j) at q (R2 + 1) + j   (odd pitch: no bank conflicts)
//   stage 2: butterfly q = t + b LPT over j < R2, gives s; element q + R1 s.
// The parity factor w_L^{p n} splits into w_L^{p j}, which joins the stage
// twiddle, and w_{2 R1}^{p r}, a compile-time constant per register (forward:
// on the inputs, n = j + R2 r; inverse: on the outputs, n = q + R1 s).
#pragma once

#include "cg_common.cuh"

namespace cg {

// ------------------------------------------------------------ constants
// cos(2 pi k / 128) for any integer k (exact decimal expansions).
__host__ __device__ constexpr double cos128(int k) {
    constexpr double tab[33] = {
        1.000000000000000000000, 0.998795456205172392714, 0.995184726672196886244, 0.989176509964780973451,
        0.980785280403230449126, 0.970031253194543992603, 0.956940335732208864935, 0.941544065183020778412,
        0.923879532511286756128, 0.903989293123443331586, 0.881921264348355029712, 0.857728610000272069902,
        0.831469612302545237078, 0.803207531480644909806, 0.773010453362736960810, 0.740951125354959091175,
        0.707106781186547524400, 0.671558954847018400625, 0.634393284163645498215, 0.595699304492433343467,
        0.555570233019602224742, 0.514102744193221726593, 0.471396736825997648556, 0.427555093430282094320,
        0.382683432365089771728, 0.336889853392220050689, 0.290284677254462367636, 0.242980179903263889948,
        0.195090322016128267848, 0.146730474455361751658, 0.098017140329560601994, 0.049067674327418014254,
        0.0};
    k &= 127;
    if (k > 64) k = 128 - k;
    return k <= 32 ? tab[k] : -tab[64 - k];
}
__host__ __device__ constexpr double sin128(int k) { return cos128(k - 32); }

// a * exp(-/+ 2 pi i K / 128) (forward / inverse)
template <int K, bool INV, typename C> __device__ __forceinline__ C mul_const(C a) {
    typedef typename real_of<C>::type R;
    if constexpr (K % 128 == 0) {
        return a;
    } else if constexpr (K == 32) {
        return INV ? mk<C>(-a.y, a.x) : mk<C>(a.y, -a.x);
    } else {
        constexpr R c = (R)cos128(K), s = (R)(INV ? sin128(K) : -sin128(K));
        return mk<C>(fma_r(a.x, c, -a.y * s), fma_r(a.x, s, a.y * c));
    }
}

// (e + w o, e - w o), w = exp(-/+ 2 pi i K / 128), 0 <= K < 64, in six fused
// multiply-adds: w o = c (o.x + (s/c) o.y, ...) with the larger of c and s
// divided out, so that the ratio stays within [-1, 1].
template <int K, bool INV, typename C> __device__ __forceinline__ void bfly(C e, C o, C &a, C &b) {
    typedef typename real_of<C>::type R;
    if constexpr (K == 0) {
        a = cadd(e, o);
        b = csub(e, o);
    } else if constexpr (K == 32) {
        const C t = mul_const<32, INV>(o);
        a = cadd(e, t);
        b = csub(e, t);
    } else {
        constexpr double c = cos128(K), s = INV ? sin128(K) : -sin128(K);
        if constexpr (K == 16 || K == 48) {
            constexpr R m = (R)c;
            // c = +-1/sqrt(2), s = +-c: w o = c (o.x - (s/c) o.y, o.y + (s/c) o.x)
            constexpr bool same = (c > 0) == (s > 0);
            const R tx = same ? o.x - o.y : o.x + o.y, ty = same ? o.y + o.x : o.y - o.x;
            a = mk<C>(fma_r(m, tx, e.x), fma_r(m, ty, e.y));
            b = mk<C>(fma_r(-m, tx, e.x), fma_r(-m, ty, e.y));
        } else if constexpr ((c < 0 ? -c : c) > (s < 0 ? -s : s)) {
            constexpr R m = (R)c, q = (R)(s / c);
            const R tx = fma_r(-q, o.y, o.x), ty = fma_r(q, o.x, o.y);
            a = mk<C>(fma_r(m, tx, e.x), fma_r(m, ty, e.y));
            b = mk<C>(fma_r(-m, tx, e.x), fma_r(-m, ty, e.y));
        } else {
            constexpr R m = (R)s, q = (R)(c / s);
            const R tx = fma_r(q, o.x, -o.y), ty = fma_r(q, o.y, o.x);
            a = mk<C>(fma_r(m, tx, e.x), fma_r(m, ty, e.y));
            b = mk<C>(fma_r(-m, tx, e.x), fma_r(-m, ty, e.y));
        }
    }
}

template <int R, int K, bool INV, typename C> __device__ __forceinline__ void wcombine(const C *e, const C *o, C *v) {
    if constexpr (K < R / 2) {
        bfly<K * (128 / R), INV>(e[K], o[K], v[K], v[K + R / 2]);
        wcombine<R, K + 1, INV>(e, o, v);
    }
}

// In-place natural-order DFT of R values in registers, unscaled.
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

// v[i] *= exp(-/+ 2 pi i I STEP / 128) for i = I .. R - 1
template <int R, int I, int STEP, bool INV, typename C> __device__ __forceinline__ void wscale(C *v) {
    if constexpr (I < R) {
        v[I] = mul_const<I * STEP, INV>(v[I]);
        wscale<R, I + 1, STEP, INV>(v);
    }
}

// ------------------------------------------------------------ plans
// Length NP = L / 2 (64 .. 256): radices, values per lane, lanes per transform,
// transforms per warp.
__host__ __device__ constexpr int wplan_r1(int NP) { return NP >= 128 ? 16 : 8; }
template <int NP> struct WPlan {
    static constexpr int R1 = wplan_r1(NP);
    static constexpr int R2 = NP / R1;
    static constexpr int E = R1;
    static constexpr int LPT = NP / E;   // lanes per transform
    static constexpr int TPW = 32 / LPT; // transforms per warp
    static constexpr int B2 = E / R2;    // stage-2 butterflies per lane (stage 1 has one: LPT = R2)
    // exchange region of one transform; several transforms of a warp start
    // LPT elements apart modulo 16, so that the 16 lanes of an 8-byte phase
    // (8 lanes of a 16-byte one) stay on distinct banks
    static constexpr int REG0 = R1 * (R2 + 1);
    static constexpr int REG = TPW == 1 ? REG0 : REG0 + ((LPT - REG0 % 16) % 16 + 16) % 16;
    static constexpr int WREG = TPW * REG;  // elements of a warp's region (>= 32 E)
    static_assert(R2 <= R1 && LPT <= 32 && WREG >= 32 * E, "two-stage plan");
};

// Twiddle tables of one (L, precision), entries exp(-2 pi i m / L), for the lane
// index l < R1 and the register index i = a + A c of stage 1's outputs:
//   forward  m = l (2 i + p):  TA[p][a][l], m = l (2 a + p);  TB[c][l], m = 2 A c l
//   inverse  m = i (2 l + p):  TA[p][a][l], m = a (2 l + p);  TB[p][c][l], m = A c (2 l + p)
// The twiddle is the product of the two entries.  Consecutive lanes read
// consecutive entries.
__host__ __device__ constexpr int wtw_base(int) { return 8; }  // A
__host__ __device__ constexpr int wtw_inv_at(int r1) { return (2 * wtw_base(r1) + r1 / wtw_base(r1)) * r1; }
__host__ __device__ constexpr int wtw_entries(int r1) {
    return wtw_inv_at(r1) + 2 * (wtw_base(r1) + r1 / wtw_base(r1)) * r1;
}
__host__ __device__ inline int wtw_exponent(int L, int r1, int i) {
    const bool inv = i >= wtw_inv_at(r1);
    if (inv) i -= wtw_inv_at(r1);
    const int l = i % r1, na = wtw_base(r1), nc = r1 / na;
    int m;
    if (i < 2 * na * r1) {
        const int p = i / (na * r1), a = (i / r1) % na;
        m = inv ? a * (2 * l + p) : l * (2 * a + p);
    } else {
        const int at = i - 2 * na * r1, p = at / (nc * r1), c = (at / r1) % nc;
        m = inv ? na * c * (2 * l + p) : 2 * na * c * l;
    }
    return m % L;
}

// v[i] *= the stage twiddle of lane l and parity p, i < R1 (conjugate for INV)
template <int R1, bool INV, typename C>
__device__ __forceinline__ void wtwiddle(C (&v)[R1], const C *__restrict__ tw, int l, int p) {
    constexpr int A = wtw_base(R1);
    const C *ta = tw + (INV ? wtw_inv_at(R1) : 0) + p * (A * R1) + l;
    const C *tb = tw + (INV ? wtw_inv_at(R1) + p * (R1 / A) * R1 : 0) + 2 * A * R1 + l;
    C wa[A];
#pragma unroll
    for (int a = 0; a < A; a++) {
        wa[a] = __ldg(ta + a * R1);
        if constexpr (INV) wa[a] = cconj(wa[a]);
        v[a] = cmul(v[a], wa[a]);
    }
#pragma unroll
    for (int c = 1; c < R1 / A; c++) {
        C wc = __ldg(tb + c * R1);
        if constexpr (INV) wc = cconj(wc);
#pragma unroll
        for (int a = 0; a < A; a++) v[A * c + a] = cmul(v[A * c + a], cmul(wa[a], wc));
    }
}

// One length-NP transform of parity p (p is uniform over the warp) in canonical
// registers: forward takes x[n] and gives X[2 m + p]; inverse takes X[2 m + p]
// and gives w_L^{-p n} IFFT_NP(...)[n].  sm: the warp's exchange region; t: lane
// within the transform; u: transform within the warp.  The region may be
// written again after __syncwarp().
template <int NP, bool INV, typename C>
__device__ __forceinline__ void wfft(C (&reg)[WPlan<NP>::E], C *sm, const C *__restrict__ tw, int t, int u, int p) {
    typedef WPlan<NP> P;
    constexpr int R1 = P::R1, R2 = P::R2, LPT = P::LPT, B2 = P::B2;
    C *x = sm + u * P::REG;
    if constexpr (!INV) {
        if (p) wscale<R1, 1, 64 / R1, false>(reg);  // w_{2 R1}^r
    }
    wdft<R1, INV>(reg);
    wtwiddle<R1, INV>(reg, tw, t, p);  // w_L^{t (2 q + p)}, inverse w_L^{-q (2 t + p)}
#pragma unroll
    for (int q = 0; q < R1; q++) x[q * (R2 + 1) + t] = reg[q];
    __syncwarp();
#pragma unroll
    for (int b = 0; b < B2; b++) {
        C v[R2];
        const int q = t + b * LPT;
#pragma unroll
        for (int j = 0; j < R2; j++) v[j] = x[q * (R2 + 1) + j];
        wdft<R2, INV>(v);
        if constexpr (INV) {
            if (p) wscale<R2, 1, 64 / R2, true>(v);  // w_{2 R2}^{-s}
        }
#pragma unroll
        for (int s = 0; s < R2; s++) reg[b + s * B2] = v[s];
    }
}

}  // namespace cg
