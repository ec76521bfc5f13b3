// Delayed-CGS2 restart cycles of small grids as one kernel.
//
// A step of the launched scheme (cg_dcgs2.cu) is six kernels.  On grids of up to
// about a hundred cells a side each of them is a few microseconds of latency: its
// launch, a chain of dependent reads of what the previous kernel wrote, a few
// hundred nanoseconds of work on a handful of SMs.  33^2 to 96^2 take 31 to 33 us
// per step, whatever the kernels' shapes.  Here one thread-block cluster of SC_CTAS
// CTAs runs the whole cycle of a system: CTA r keeps its rows of u and w in shared
// memory, the transforms exchange rows and columns through distributed shared
// memory, and three cluster barriers replace the six launches of a step:
//
//   rows forward   -> every column's owner                     barrier
//   columns        -> every row's owner                        barrier
//   rows inverse: w = A u; partial dots with the basis          barrier
//   every CTA adds the partial sums (same order, so the same values), forms the
//   step's coefficients, rotations and stop decision for itself, and updates its
//   rows of q_k and u_{k+1}; CTA 0 writes what the rest of the solve reads.
//
// A step at 64^2 with 25 vectors: rows 1.5, columns 2.0, rows 1.1, dots 2.6, sums
// 0.8, step 2.3, update 2.2, t_k 0.8 us.  The basis streams from L2 into 16 SMs
// instead of all of them, which is the price: it ends the gain on larger grids.
// Whole FP64 solves of up to 100 steps, us per step, launched / one kernel: 33^2
// 32.2 / 15.9, 48^2 32.8 / 16.4, 64^2 33.8 / 17.5; the same kernel built for L = 256:
// 65^2 31.1 / 26.5, 80^2 32.1 / 32.5, 96^2 32.8 / 35.5, 112^2 33.2 / 46.  Only L = 128 (33 <=
// N <= 64) is built; the sides from 65 to 79 that L = 256 would serve faster are launched.
// A bucket of systems runs one cluster per system.
//
// Transforms: cg_wfft.cuh, NP = L / 2 = 64, four per warp; a pair of warps takes
// the two parities of four lines.
#include <cooperative_groups.h>
#include <stdlib.h>

#include <type_traits>

#include "cg_internal.h"
#include "cg_wfft.cuh"

namespace cg {

namespace {

namespace cgr = cooperative_groups;

constexpr int SC_CTAS = 16, SC_THREADS = 256, SC_WARPS = SC_THREADS / 32;
constexpr int NP = WPlan::NP;

// Shared memory of one CTA, in bytes from the start.
struct SmallSmem {
    int su, sw, sc, tb, rb, ex, part, d1, d2, tv, cs, sn, col, pc, bytes;
};
template <typename C> __host__ __device__ constexpr SmallSmem small_smem(int N, int m) {
    typedef WPlan P;
    const int rpc = (N + SC_CTAS - 1) / SC_CTAS, ns = rpc * N, e = sizeof(C);
    SmallSmem s{};
    int o = 0;
    auto take = [&](int bytes) {
        const int at = o;
        o += (bytes + 15) / 16 * 16;
        return at;
    };
    s.su = take(ns * e);
    s.sw = take(ns * e);
    s.sc = take(ns * e / 2);
    s.tb = take(2 * NP / SC_CTAS * (N + 1) * e);
    s.rb = take(rpc * (2 * NP + 1) * e);
    s.ex = take(SC_WARPS * P::WREG * e);
    s.part = take(4 * (m + 2) * 8);
    s.d1 = take((m + 2) * 16);
    s.d2 = take((m + 2) * 16);
    s.tv = take(2 * (m + 2) * 16);
    s.cs = take((m + 1) * 16);
    s.sn = take((m + 1) * 8);
    s.col = take((m + 2) * 16);
    s.pc = take(2 * (m + 2) * e);  // P and S of the axpy
    s.bytes = o;
    return s;
}

__device__ __forceinline__ void pair_sync(int pair) { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); }

// Adds the partner's parity to one half of the line (see cg_wfft.cuh: warp p of a
// pair ends with values [p E/2, (p + 1) E/2)): out(i, value) for each.
template <int P, int E, typename C, typename F>
__device__ __forceinline__ void join_half(const C (&reg)[E], C *mine, const C *other, int lane, int pair, F out) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < E / 2; i++) mine[i * 32 + lane] = reg[P ? i : i + E / 2];
    pair_sync(pair);
#pragma unroll
    for (int i = 0; i < E / 2; i++) out(i + P * (E / 2), cadd(reg[i + P * (E / 2)], other[i * 32 + lane]));
}

// Sum of four values over the warp: lane 8 q holds the total of a_q.
__device__ __forceinline__ double sum4(double a0, double a1, double a2, double a3, int lane) {
    const bool b4 = lane & 16, b3 = lane & 8;
    const double s0 = b4 ? a0 : a2, s1 = b4 ? a1 : a3;
    const double k0 = (b4 ? a2 : a0) + __shfl_xor_sync(0xffffffffu, s0, 16);
    const double k1 = (b4 ? a3 : a1) + __shfl_xor_sync(0xffffffffu, s1, 16);
    double m = (b3 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, b3 ? k0 : k1, 8);
    m += __shfl_xor_sync(0xffffffffu, m, 4);
    m += __shfl_xor_sync(0xffffffffu, m, 2);
    m += __shfl_xor_sync(0xffffffffu, m, 1);
    return m;
}

// conj(a) u and conj(a) w added to four FP64 sums; FP32 products are exact in FP64
template <typename C> __device__ __forceinline__ void dot2(C a, C u, C w, double (&s)[4]) {
    const double ax = a.x, ay = a.y, ux = u.x, uy = u.y, wx = w.x, wy = w.y;
    s[0] = fma(ax, ux, fma(ay, uy, s[0]));
    s[1] = fma(ax, uy, fma(-ay, ux, s[1]));
    s[2] = fma(ax, wx, fma(ay, wy, s[2]));
    s[3] = fma(ax, wy, fma(-ay, wx, s[3]));
}

// One CTA's share of the operator: the arrays, and this lane's place in them.
template <typename C> struct SmallOp {
    typedef typename real_of<C>::type R;
    typedef WPlan P;
    static constexpr int E = P::E, LPT = P::LPT, TPW = P::TPW, CPC = 2 * NP / SC_CTAS;
    static_assert(TPW == 4 && CPC % TPW == 0 && CPC / TPW * 2 <= SC_WARPS, "a warp pair per four columns");
    C *su, *sw, *tb, *rb, *mine;
    const C *other, *twl;
    R *sc;
    int N, rank, rpc, r0, rows, ns, ldt, ldr, lane, pair, p, t, u4, c_loc, transpose;
    bool has_col;
    C gv[E];  // this lane's spectrum values: column c_loc of the CTA, rows 2 (t + i LPT) + p

    __device__ __forceinline__ SmallOp(unsigned char *smem, const SmallSmem &lay, int N_, int rank_, const C *gq, const C *tw,
                                       int transpose_) {
        N = N_, rank = rank_, transpose = transpose_;
        const int warp = threadIdx.x >> 5;
        lane = threadIdx.x & 31, pair = warp >> 1, p = warp & 1, t = lane % LPT, u4 = lane / LPT;
        su = reinterpret_cast<C *>(smem + lay.su), sw = reinterpret_cast<C *>(smem + lay.sw);
        sc = reinterpret_cast<R *>(smem + lay.sc);
        tb = reinterpret_cast<C *>(smem + lay.tb), rb = reinterpret_cast<C *>(smem + lay.rb);
        mine = reinterpret_cast<C *>(smem + lay.ex) + warp * P::WREG;
        other = reinterpret_cast<C *>(smem + lay.ex) + (warp ^ 1) * P::WREG;
        twl = tw + 8 * NP;  // tables of cg_wfft.cuh follow the 4 L entries of cg_fft.cuh
        rpc = (N + SC_CTAS - 1) / SC_CTAS, r0 = rank * rpc;
        rows = r0 >= N ? 0 : N - r0 < rpc ? N - r0 : rpc;
        ns = rows * N, ldt = N + 1, ldr = 2 * NP + 1;
        c_loc = pair * TPW + u4;
        has_col = pair * TPW < CPC;
        if (has_col) {
            const int m = rank * CPC + c_loc, h = m / NP, kc = 2 * (m % NP) + h, qc = kc <= NP ? kc : 2 * NP - kc;
#pragma unroll
            for (int i = 0; i < E; i++) {
                const int k1 = 2 * (t + i * LPT) + p, qr = k1 <= NP ? k1 : 2 * NP - k1;
                gv[i] = gq[(size_t)qc * (NP + 1) + qr];
            }
        }
    }

    // sw = A su (A^T su with transpose).  Two cluster barriers: the caller's CTAs are
    // all inside, with su and sc written (__syncthreads), and none of them may still
    // read tb or rb of the previous application, which one more cluster barrier
    // between two calls ensures.
    __device__ __forceinline__ void apply(cgr::cluster_group &cl) {
        // ------------------------------------------------ rows forward, to the columns' owners
        const bool row_warp = pair * TPW < rows;
        const int rl = pair * TPW + u4;
        if (row_warp) {
            C reg[E];
#pragma unroll
            for (int i = 0; i < E; i++) {
                const int x = t + i * LPT;
                reg[i] = czero<C>();
                if (rl < rows && x < N) reg[i] = transpose ? su[rl * N + x] : cscale(su[rl * N + x], sc[rl * N + x]);
            }
            wfft<false>(reg, mine, twl, t, u4, p);
            if (rl < rows) {
#pragma unroll
                for (int i = 0; i < E; i++) {
                    const int c = p * NP + t + i * LPT;
                    cl.map_shared_rank(tb, c / CPC)[(c % CPC) * ldt + r0 + rl] = reg[i];
                }
            }
        }
        cl.sync();
        // ------------------------------------------------ columns, to the rows' owners
        if (has_col) {
            C reg[E];
#pragma unroll
            for (int i = 0; i < E; i++) {
                const int y = t + i * LPT;
                reg[i] = y < N ? tb[c_loc * ldt + y] : czero<C>();
            }
            wfft<false>(reg, mine, twl, t, u4, p);
#pragma unroll
            for (int i = 0; i < E; i++) reg[i] = cmul(reg[i], gv[i]);
            __syncwarp();
            wfft<true>(reg, mine, twl, t, u4, p);
            auto put = [&](int i, C v) {
                const int y = t + i * LPT;
                if (y < N) cl.map_shared_rank(rb, y / rpc)[(y % rpc) * ldr + rank * CPC + c_loc] = v;
            };
            if (p) join_half<1>(reg, mine, other, lane, pair, put);
            else join_half<0>(reg, mine, other, lane, pair, put);
        }
        cl.sync();
        // ------------------------------------------------ rows inverse: w = u - G c u (or u - c G u)
        if (row_warp) {
            C reg[E];
#pragma unroll
            for (int i = 0; i < E; i++) reg[i] = rl < rows ? rb[rl * ldr + p * NP + t + i * LPT] : czero<C>();
            wfft<true>(reg, mine, twl, t, u4, p);
            auto put = [&](int i, C v) {
                const int x = t + i * LPT;
                if (rl < rows && x < N) {
                    if (transpose) v = cscale(v, sc[rl * N + x]);
                    sw[rl * N + x] = csub(su[rl * N + x], v);
                }
            };
            if (p) join_half<1>(reg, mine, other, lane, pair, put);
            else join_half<0>(reg, mine, other, lane, pair, put);
        }
        __syncthreads();
    }
};

template <typename C>
__global__ void __launch_bounds__(SC_THREADS, 1)
k_small_cycle(C *V, long long n, KrylovPtrs kp, int N, const typename real_of<C>::type *cdiag, const C *gq,
              const C *__restrict__ tw, int transpose, int m, long long sys_c, long long sys_gq) {
    typedef typename real_of<C>::type R;
    kp = kp_sys(kp);
    V = sys_vec(V, kp);
    cdiag += (long long)blockIdx.y * sys_c;
    gq += (long long)blockIdx.y * sys_gq;
    DevState *st = kp.st;
    if (st->stop) return;  // the whole cluster
    cgr::cluster_group cl = cgr::this_cluster();
    const int rank = (int)cl.block_rank();
    extern __shared__ __align__(16) unsigned char smem[];
    const SmallSmem lay = small_smem<C>(N, m);
    double *part = reinterpret_cast<double *>(smem + lay.part);
    double2 *D1 = reinterpret_cast<double2 *>(smem + lay.d1), *D2 = reinterpret_cast<double2 *>(smem + lay.d2);
    double2 *tvs = reinterpret_cast<double2 *>(smem + lay.tv), *css = reinterpret_cast<double2 *>(smem + lay.cs);
    double *sns = reinterpret_cast<double *>(smem + lay.sn);
    double2 *col = reinterpret_cast<double2 *>(smem + lay.col);
    C *Pc = reinterpret_cast<C *>(smem + lay.pc), *Sc = Pc + (m + 2);
    __shared__ double red[SC_WARPS][4];
    __shared__ double scan_a[SC_THREADS];
    __shared__ double2 scan_b[SC_THREADS];
    __shared__ double2 carry_last;
    __shared__ double2 fin_gk;  // g_k of the rotated right-hand side
    __shared__ int fin_stop;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    SmallOp<C> op(smem, lay, N, rank, gq, tw, transpose);
    C *su = op.su, *sw = op.sw;
    const int ns = op.ns;
    const size_t base = (size_t)op.r0 * N;
    for (int e = tid; e < ns; e += SC_THREADS) {
        su[e] = V[base + e];
        op.sc[e] = cdiag[base + e];
    }
    const int m_max = st->m < m ? st->m : m, maxit = st->maxit, ref = st->rotation == 1, fixed = st->fixed, ld = kp.mcap + 1;
    const double tol_abs = st->tol * st->nb, inner_abs = st->inner_tol * st->beta0, nb = st->nb;
    int it = st->it;
    __syncthreads();
    cl.sync();  // every CTA's shared memory may be written from here on

    for (int k = 0;; k++) {
        op.apply(cl);
        // ------------------------------------------------ partial dots with q_0 .. q_{k-1} and u
        constexpr int DU = 4;  // 16 loads in flight a lane
        for (int j0 = 4 * warp; j0 < k; j0 += 4 * SC_WARPS) {
            double s[4][4] = {};
            const C *v0 = V + (size_t)j0 * n + base;
            const int nj = k - j0 < 4 ? k - j0 : 4;
            for (int e0 = lane; e0 < ns; e0 += 32 * DU) {
                C a[DU][4];
#pragma unroll
                for (int r = 0; r < DU; r++)
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        a[r][q] = e0 + 32 * r < ns ? __ldcg(v0 + (size_t)(q < nj ? q : 0) * n + e0 + 32 * r) : czero<C>();
#pragma unroll
                for (int r = 0; r < DU; r++) {
                    const int e = e0 + 32 * r < ns ? e0 + 32 * r : 0;
                    const C uu = su[e], ww = sw[e];
#pragma unroll
                    for (int q = 0; q < 4; q++) dot2(a[r][q], uu, ww, s[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const double d = sum4(s[q][0], s[q][1], s[q][2], s[q][3], lane);
                if (q < nj && (lane & 7) == 0) part[4 * (j0 + q) + (lane >> 3)] = d;
            }
        }
        if (warp == SC_WARPS - 1) {
            double s[4] = {};
            for (int e = lane; e < ns; e += 32) dot2(su[e], su[e], sw[e], s);
            const double d = sum4(s[0], s[1], s[2], s[3], lane);
            if ((lane & 7) == 0) part[4 * k + (lane >> 3)] = d;
        }
        cl.sync();
        // ------------------------------------------------ sums over the CTAs, in rank order
        for (int q = tid; q < 4 * (k + 1); q += SC_THREADS) {
            double v[SC_CTAS], s = 0.0;
#pragma unroll
            for (int r = 0; r < SC_CTAS; r++) v[r] = cl.map_shared_rank(part, r)[q];
#pragma unroll
            for (int r = 0; r < SC_CTAS; r++) s += v[r];
            reinterpret_cast<double *>(((q & 3) < 2 ? D1 : D2) + (q >> 2))[q & 1] = s;
        }
        __syncthreads();
        // ------------------------------------------------ the step, as in dcgs2_step (every CTA the same)
        const double2 *tv = tvs + (k & 1) * (m + 2);
        double sa = 0.0, acr = 0.0, aci = 0.0, hn = 0.0;
        for (int j = tid; j < k; j += SC_THREADS) {
            const double2 a = D1[j], c = D2[j];
            sa += a.x * a.x + a.y * a.y;
            acr += a.x * c.x + a.y * c.y;  // conj(a) c
            aci += a.x * c.y - a.y * c.x;
            const double2 h = cadd(tv[j], a);  // column k-1 of H above the subdiagonal
            hn += h.x * h.x + h.y * h.y;
            col[j] = h;
        }
        sa = warp_sum(sa);
        acr = warp_sum(acr);
        aci = warp_sum(aci);
        hn = warp_sum(hn);
        if (lane == 0) red[warp][0] = sa, red[warp][1] = acr, red[warp][2] = aci, red[warp][3] = hn;
        __syncthreads();
        sa = acr = aci = hn = 0.0;
#pragma unroll
        for (int w = 0; w < SC_WARPS; w++) sa += red[w][0], acr += red[w][1], aci += red[w][2], hn += red[w][3];
        const double alpha = D1[k].x;
        const double2 d = D2[k];
        double nu2 = alpha - sa;
        if (!isfinite(nu2) || !isfinite(acr) || !isfinite(aci) || !isfinite(d.x) || !isfinite(d.y) || !isfinite(hn)) {
            if (rank == 0 && tid == 0) {
                st->status = 4;
                st->stop = 1;
            }
            break;
        }
        if (!(nu2 > 0.0)) nu2 = 0.0;
        const bool brk = k >= 1 ? !(nu2 > 1e-28 * (hn + nu2)) : !(nu2 > 0.0);
        const double nu = sqrt(nu2), inu = nu > 0.0 ? 1.0 / nu : 0.0;
        const double2 delta = make_double2((d.x - acr) * inu, (d.y - aci) * inu);
        if (k >= 1) {
            if (rank == 0)
                for (int i = tid; i < k; i += SC_THREADS) kp.Hm[(size_t)i * ld + (k - 1)] = col[i];
            if (tid == 0) {
                col[k] = make_double2(nu, 0.0);
                if (rank == 0) kp.Hm[(size_t)k * ld + (k - 1)] = make_double2(nu, 0.0);
            }
        }
        for (int i = tid; i < k; i += SC_THREADS) {
            const double2 a = D1[i], c = D2[i], da = cmul(delta, a);
            Pc[i] = mk<C>((R)(a.x * inu), (R)(a.y * inu));
            Sc[i] = mk<C>((R)((c.x - da.x * inu) * inu), (R)((c.y - da.y * inu) * inu));
        }
        // rotations 0..k-2 applied to col[0..k-1] by a prefix scan of affine maps
        if (k >= 1) {
            const int nr = k - 1, seg = (nr + SC_THREADS - 1) / SC_THREADS;
            const int j0 = tid * seg < nr ? tid * seg : nr, j1 = j0 + seg < nr ? j0 + seg : nr;
            double a = 1.0;
            double2 b = make_double2(0.0, 0.0);
            for (int j = j0; j < j1; j++) {
                a = -sns[j] * a;
                b = cadd(cscale(b, -sns[j]), cmul(css[j], col[j + 1]));
            }
            scan_a[tid] = a;
            scan_b[tid] = b;
            __syncthreads();
            for (int off = 1; off < SC_THREADS && off < nr; off <<= 1) {
                const double a2 = scan_a[tid], a1 = tid >= off ? scan_a[tid - off] : 1.0;
                const double2 b2 = scan_b[tid], b1 = tid >= off ? scan_b[tid - off] : make_double2(0.0, 0.0);
                __syncthreads();
                if (tid >= off) {
                    scan_a[tid] = a2 * a1;
                    scan_b[tid] = cadd(cscale(b1, a2), b2);
                }
                __syncthreads();
            }
            double2 carry = col[0];
            if (tid > 0) carry = cadd(cscale(col[0], scan_a[tid - 1]), scan_b[tid - 1]);
            for (int j = j0; j < j1; j++) {
                const double2 nx = col[j + 1], c = css[j];
                if (rank == 0)
                    kp.Rm[(size_t)(k - 1) * ld + j] = cadd(cmul(ref ? c : cconj(c), carry), cscale(nx, sns[j]));
                carry = csub(cmul(c, nx), cscale(carry, sns[j]));
            }
            if (nr == 0 ? tid == 0 : (j0 < j1 && j1 == nr)) carry_last = carry;
        }
        __syncthreads();
        if (tid == 0) {
            int stop = 0;
            if (k == 0) {
                fin_gk = make_double2(nu, 0.0);
                if (rank == 0) kp.g[0] = fin_gk;
            } else {
                const double2 carry = carry_last;
                const double rho = hypot(hypot(carry.x, carry.y), nu);
                double2 c = make_double2(1.0, 0.0);
                double s = 0.0;
                if (rho > 0.0 && isfinite(rho)) {
                    c = make_double2(carry.x / rho, carry.y / rho);
                    s = nu / rho;
                }
                const double2 cc = ref ? c : cconj(c), gk = fin_gk;
                css[k - 1] = c;
                sns[k - 1] = s;
                fin_gk = cscale(gk, -s);
                const double gabs = hypot(gk.x, gk.y) * s;
                if (!fixed && (gabs <= tol_abs || gabs <= inner_abs)) stop = 1;
                if (k >= m_max || it + 1 >= maxit) stop = 1;
                if (rank == 0) {
                    kp.Rm[(size_t)(k - 1) * ld + (k - 1)] = cadd(cmul(cc, carry), make_double2(s * nu, 0.0));
                    kp.cs[k - 1] = c;
                    kp.sn[k - 1] = s;
                    kp.g[k] = fin_gk;
                    kp.g[k - 1] = cmul(cc, gk);
                    kp.hist[it + 1] = gabs / nb;
                    st->it = it + 1;
                    st->est = gabs / nb;
                    st->ncol = k;
                }
            }
            if (brk) stop = 1;
            fin_stop = stop;
            if (rank == 0) {
                if (brk) st->brk = 1;
                st->k = k + 1;
                st->stop = stop;
            }
        }
        __syncthreads();
        if (k >= 1) it++;
        if (fin_stop) break;
        // ------------------------------------------------ q_k and u_{k+1} on this CTA's rows
        const R cu = (R)inu, cw = (R)inu;
        const C du = mk<C>((R)(-delta.x * inu * inu), (R)(-delta.y * inu * inu));
        for (int e = tid; e < ns; e += SC_THREADS) {
            // U loads in flight a thread.  Each U vectors are summed apart, in two chains: one
            // chain of k rounded sums loses more than the launched pass's eight of k / 8
            // (complex64, relative rms in units of 2^-24 at k = 25 / 100 / 400 / 1200: eight chains
            // 1.16 / 1.43 / 2.30 / 3.8, one 1.50 / 2.93 / 5.96 / 10.5, these 1.02 / 1.31 / 1.87 / 2.8).
            constexpr int U = 16;
            C s1 = czero<C>(), s2 = czero<C>();
            const C *v = V + base + e;
            for (int j0 = 0; j0 < k; j0 += U) {
                C a[U], p1[2] = {czero<C>(), czero<C>()}, p2[2] = {czero<C>(), czero<C>()};
#pragma unroll
                for (int q = 0; q < U; q++) a[q] = j0 + q < k ? __ldcg(v + (size_t)(j0 + q) * n) : czero<C>();
#pragma unroll
                for (int q = 0; q < U; q++) {
                    if (j0 + q >= k) break;
                    p1[q & 1] = cfma(p1[q & 1], Pc[j0 + q], a[q]);
                    p2[q & 1] = cfma(p2[q & 1], Sc[j0 + q], a[q]);
                }
                s1 = cadd(s1, cadd(p1[0], p1[1]));
                s2 = cadd(s2, cadd(p2[0], p2[1]));
            }
            const C uu = su[e], ww = sw[e];
            V[(size_t)k * n + base + e] = csub(cscale(uu, cu), s1);
            su[e] = csub(cadd(cscale(ww, cw), cmul(du, uu)), s2);
        }
        // t_k = ([c; delta] - H(0:k, 0:k-1) a) / nu, a warp per row, rows dealt to the CTAs, to every CTA's next buffer
        // (column k-1 of H is the one in col; the earlier ones were written before the last barriers)
        double2 *tn = tvs + ((k + 1) & 1) * (m + 2);
        for (int i = rank + SC_CTAS * warp; i <= k; i += SC_CTAS * SC_WARPS) {
            double er = 0.0, ei = 0.0;
            for (int j = (i > 0 ? i - 1 : 0) + lane; j < k; j += 32) {
                const double2 h = j == k - 1 ? col[i] : __ldcg(kp.Hm + (size_t)i * ld + j);
                const double2 a = D1[j];
                er += h.x * a.x - h.y * a.y;
                ei += h.x * a.y + h.y * a.x;
            }
            er = warp_sum(er);
            ei = warp_sum(ei);
            const double2 c = i < k ? D2[i] : delta;
            if (lane < SC_CTAS) cl.map_shared_rank(tn, lane)[i] = make_double2((c.x - er) * inu, (c.y - ei) * inu);
        }
        __syncthreads();
    }
    cl.sync();  // no CTA leaves while another may still read or write its shared memory
}

// y = A x (A^T x) as one launch.
template <typename C>
__global__ void __launch_bounds__(SC_THREADS, 1)
k_small_matvec(const C *x, C *y, int N, const typename real_of<C>::type *cdiag, const C *gq, const C *__restrict__ tw,
               int transpose) {
    cgr::cluster_group cl = cgr::this_cluster();
    extern __shared__ __align__(16) unsigned char smem[];
    SmallOp<C> op(smem, small_smem<C>(N, 0), N, (int)cl.block_rank(), gq, tw, transpose);
    const size_t base = (size_t)op.r0 * N;
    for (int e = threadIdx.x; e < op.ns; e += SC_THREADS) {
        op.su[e] = x[base + e];
        op.sc[e] = cdiag[base + e];
    }
    __syncthreads();
    cl.sync();  // every CTA's shared memory may be written from here on
    op.apply(cl);
    for (int e = threadIdx.x; e < op.ns; e += SC_THREADS) y[base + e] = op.sw[e];
}

cudaLaunchConfig_t cluster_config(int nsys, int bytes, cudaLaunchAttribute *at, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(SC_CTAS, nsys);
    cfg.blockDim = dim3(SC_THREADS);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = SC_CTAS;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}
// 220 KB: a CTA's shared memory (227 KB) less these kernels' static arrays.  Always
// the same limit, whatever the launch needs (see smem_optin, whose look at the
// kernel would add 0.4 us to the 26 of a product that is waited for).
constexpr int SC_SMEM = 220 * 1024;
template <typename K> int cluster_optin(K kern) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SC_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return (int)e;
}

template <typename C>
int launch(void *V, long long n, const KrylovPtrs &kp, int m, const MatvecArgs &a, cudaStream_t s) {
    typedef typename real_of<C>::type R;
    auto kern = k_small_cycle<C>;
    const int bytes = small_smem<C>(a.N, m).bytes;
    if (int e = cluster_optin(kern)) return e;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cluster_config(kp.nsys, bytes, &at, s);
    return (int)cudaLaunchKernelEx(&cfg, kern, (C *)V, n, kp, a.N, (const R *)a.cdiag, (const C *)a.gq,
                                   (const C *)a.tw, a.transpose, m, a.sys_c, a.sys_gq);
}
template <typename C> int launch_mv(const void *x, void *y, const MatvecArgs &a, cudaStream_t s) {
    typedef typename real_of<C>::type R;
    auto kern = k_small_matvec<C>;
    const int bytes = small_smem<C>(a.N, 0).bytes;
    if (int e = cluster_optin(kern)) return e;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cluster_config(1, bytes, &at, s);
    return (int)cudaLaunchKernelEx(&cfg, kern, (const C *)x, (C *)y, a.N, (const R *)a.cdiag, (const C *)a.gq,
                                   (const C *)a.tw, a.transpose);
}

template <typename C> bool fits(int N, int m) {
    static const int most = [] {  // clusters that the device holds at that size
        auto kern = k_small_cycle<C>;
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t cfg = cluster_config(1, SC_SMEM, &at, nullptr);
        int c = 0;
        if (cluster_optin(kern) != 0 || cudaOccupancyMaxActiveClusters(&c, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            c = 0;
        }
        return c;
    }();
    return most > 0 && small_smem<C>(N, m).bytes <= SC_SMEM;
}

}  // namespace

int small_cycle_fits(int prec, int N, int L, int m) {
    // CUGMRES_SMALL_CYCLE=0, or a forced shape of the launched passes: diagnostics
    static const bool on = [] {
        const char *e = getenv("CUGMRES_SMALL_CYCLE");
        if (e && e[0] == '0') return false;
        for (const char *v : {"CUGMRES_DOTS2_SHAPE", "CUGMRES_AXPY2_SHAPE", "CUGMRES_MATVEC_SHAPE"}) {
            const char *f = getenv(v);
            if (f && *f) return false;
        }
        return true;
    }();
    if (!on || L != WPlan::L) return 0;
    return prec == 0 ? fits<double2>(N, m) : fits<float2>(N, m);
}

int launch_small_cycle(int prec, void *V, long long n, const KrylovPtrs &kp, int m, const MatvecArgs &a, cudaStream_t s) {
    if (a.L != WPlan::L || m > kp.mcap) return (int)cudaErrorInvalidValue;
    return prec == 0 ? launch<double2>(V, n, kp, m, a, s) : launch<float2>(V, n, kp, m, a, s);
}

int launch_small_matvec(int prec, const void *x, void *y, const MatvecArgs &a, cudaStream_t s) {
    if (a.L != WPlan::L) return (int)cudaErrorInvalidValue;
    return prec == 0 ? launch_mv<double2>(x, y, a, s) : launch_mv<float2>(x, y, a, s);
}

}  // namespace cg
