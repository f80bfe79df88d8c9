// Scalar Legendre kernels in FP64 (the FP32 ones are in hb_legendre32.cu).
//
// Replaces the reference's per-m pipeline (sht_raw.py:46-56: one plm_recurrence launch per m
// writing the [Nr, lmax+1] Lambda block to HBM (legendre.cu:2-35), host-side factorial norms
// (sht_raw.py:26-28, which overflow above lmax 85), a per-ring host gather of F_r[m] and a
// per-l scatter) and the synthesis loops of isht.py:11-23.
//
// Lambda is generated in registers and never stored.  Equatorial symmetry folds the north and
// south rings of a pair into E = F_N + F_S (even l-m) and O = F_N - F_S (odd l-m).  With
// eps_l = sqrt((l^2-m^2)/(4l^2-1)), x lambda_l = eps_{l+1} lambda_{l+1} + eps_l lambda_{l-1}, so the
// functions r_k = lambda_{m+2k+1} / x carry both parities (Ishioka 2018, J. Meteor. Soc. Japan 96):
//     lambda_{l+1} = x r_k,   lambda_l = eps_{l+1} r_k + eps_l r_{k-1}      (l = m + 2k),
// and one recursion over k serves two l.  Scaled to r_k = N_k rho_k with
// N_k N_{k+1} eps_{l+2} eps_{l+3} = 1/4 its last coefficient is 1; with s = sin theta and
// alpha_k = 4 N_k^2 it runs on the difference d_k = rho_k - rho_{k-1},
//     rho_k = rho_{k-1} + d_k,   d_{k+1} = d_k + (gamma_k - alpha_k s^2) rho_k,
//     gamma_k = alpha_k (1 - eps_{l+1}^2 - eps_{l+2}^2) - 2,
// which keeps its accuracy towards the poles, where rho varies slowly (Reinsch's form): 3
// operations for two l and 4 per map for the contraction, against 6 and 4 in the one-step form
// lambda_l = A x lambda_{l-1} + B lambda_{l-2}.  r_k grows like 1/x, so rings near the equator
// (|x| < LEG_X0) use the one-step recursion, scaled the same way, lambda_l = M_l y_l,
// M_l M_{l+1} eps_{l+1} = 1/2: y_{l+1} = 2 M_l^2 x y_l - y_{l-1}, 4 operations for two l (signs of
// period 4 absorbed in the tables turn the subtraction into an addition).
// Error against an independent 64-bit reference (alm2map, map2alm at nside 1024, lmax 2047): 3.3e-14,
// 4.8e-14 (one-step form: 3.3e-14, 5.1e-14; with LEG_X0 = 0.3 instead of 0.5 it is 3.6e-14, 5.4e-14, at
// 1 % less time).
//
// The coefficients are tables of the plan (LegTab).  Start values come from log2 tables, carried as
// mantissa * 2^(512 e): while e < 0 a value is below 2^-256, and the state is rescaled whenever it
// passes 2^256, so nothing overflows or underflows up to lmax = 16383.
//
// What bounds the kernels: the FP64 pipe (62 FMA per clock and SM measured); the analysis adds a
// warp reduction per l.  One map at nside 1024, lmax 2047: synthesis 2063 -> 1160 us, analysis
// 2826 -> 1680 us (one-step form with a shared-memory reduction per l before); two maps 1.8 times one.
#include <cmath>

#include "hb_internal.cuh"
#include "hb_warp.cuh"

namespace hb {

constexpr int LKB = 128;  // two-l steps per staged block of 256 l

// start value lambda_mm = mant * 2^(512 e)
__device__ __forceinline__ void sectoral_start64(const GeomDev &g, int m, int64_t p, double &mant, int &e) {
    const double L = g.log2cm[m] + (double)m * g.pair_log2sin[p];
    e = (int)floor((L + 256.0) / 512.0);
    const double v = exp2(L - 512.0 * e);
    mant = (m & 1) ? -v : v;
}

// Recursion zones (see the file comment)
enum { ZPOLE = 0, ZEQ = 1 };

// U ring pairs per lane of one warp: pair 32 (grp U + u) + lane
// ZPOLE: r = rho_{k-1}, d = d_k, w = -s^2.  ZEQ: r = y_{l-1}, d = y_{l-2}, w = x.
template <int U> struct State {
    double r[U], d[U], w[U];
    int e[U];
};
template <int U> __device__ __forceinline__ int64_t unit_pair(int grp, int u, int lane) {
    return (int64_t)(grp * U + u) * 32 + lane;
}

// ring positions and start values of a group; returns its zone
template <int U> __device__ __forceinline__ int start_group(const GeomDev &g, const double *tab, int m, int grp, int lane, State<U> &S) {
    double x[U];
    bool pole = true;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t p = unit_pair<U>(grp, u, lane);
        x[u] = p < g.npairs ? g.pair_x[p] : 0.0;
        if (p < g.npairs) pole &= x[u] >= LEG_X0;
    }
    const int zone = __all_sync(0xffffffffu, pole) ? ZPOLE : ZEQ;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t p = unit_pair<U>(grp, u, lane);
        S.w[u] = zone == ZPOLE ? (x[u] - 1.0) * (x[u] + 1.0) : x[u];
        S.r[u] = S.d[u] = 0.0;
        S.e[u] = 0;
        if (p < g.npairs) {  // rho_0 = lambda_mm / (N_0 eps_{m+1}), y_m = lambda_mm / M_m
            double mant;
            sectoral_start64(g, m, p, mant, S.e[u]);
            S.d[u] = mant / (zone == ZPOLE ? tab[LT_P] : tab[LT_M0]);
        }
    }
    return zone;
}

// one two-l step; f(u, even value, odd value) sees (rho, rho) in ZPOLE
template <int ZONE, int U, typename Fn> __device__ __forceinline__ void two_step(State<U> &S, double2 c, Fn f) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (ZONE == ZPOLE) {
            S.r[u] += S.d[u];
            f(u, S.r[u], S.r[u]);
            S.d[u] = fma(fma(c.x, S.w[u], c.y), S.r[u], S.d[u]);
        } else {
            S.d[u] = fma(c.x * S.w[u], S.r[u], S.d[u]);
            S.r[u] = fma(c.y * S.w[u], S.d[u], S.r[u]);
            f(u, S.d[u], S.r[u]);
        }
    }
}

enum { CLEAN = 0, MIXED = 1, DEAD = 2 };  // no / some / every value of the warp's group has e < 0

template <int U> __device__ __forceinline__ int mode_of(const State<U> &S) {
    bool neg = false, live = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        neg |= S.e[u] < 0;
        live |= S.e[u] >= 0;
    }
    if (!__any_sync(0xffffffffu, neg)) return CLEAN;
    return __any_sync(0xffffffffu, live) ? MIXED : DEAD;
}

// Brings values that have grown past 2^256 to the next exponent; up(u) is told of each.  False when
// the warp has none (one vote, the usual case).
template <int U, typename Fn> __device__ __forceinline__ bool rescale(State<U> &S, Fn up) {
    bool any = false;
#pragma unroll
    for (int u = 0; u < U; ++u) any |= S.e[u] < 0 && fabs(S.r[u]) > 0x1p256;
    if (!__any_sync(0xffffffffu, any)) return false;
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (S.e[u] < 0 && fabs(S.r[u]) > 0x1p256) {
            S.r[u] *= 0x1p-512;
            S.d[u] *= 0x1p-512;
            ++S.e[u];
            up(u);
        }
    return true;
}

// four consecutive table values (rows are 16-byte aligned)
__device__ __forceinline__ double4 four(const double *t) {
    const double2 a = *reinterpret_cast<const double2 *>(t), b = *reinterpret_cast<const double2 *>(t + 2);
    return make_double4(a.x, a.y, b.x, b.y);
}

// ------------------------------------------------------------------ analysis
template <int NB, int U> struct Weights {
    double er[NB][U], ei[NB][U], qr[NB][U], qi[NB][U];
};

// TL two-l steps: values times weights summed over the group's pairs, added to the warp's row
// red[(step * NB + map) * 4 + (E re, E im, O re, O im)].  GATED: pairs with e < 0 take no part.  Their terms are
// predicated off: a zero value in their place would turn an infinite or NaN weight into NaN, and costs more
// (nside 1024, lmax 2047: one map 1680 us, 1705 with zeroed values; two 3021, 3082).
template <int ZONE, bool GATED, int U, int NB, int TL>
__device__ __forceinline__ void anal_chunk(State<U> &S, const Weights<NB, U> &W, const double2 *cf, double *red, int lane) {
    double v[TL * NB * 4];
#pragma unroll
    for (int s = 0; s < TL; ++s) {
        two_step<ZONE>(S, cf[s], [&](int u, double ve, double vo) {
            if (GATED) {
#pragma unroll
                for (int i = 0; i < NB * 4; ++i)
                    if (u == 0) v[s * NB * 4 + i] = 0.0;
                if (S.e[u] >= 0) {
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        double *a = v + (s * NB + b) * 4;
                        a[0] = fma(ve, W.er[b][u], a[0]);
                        a[1] = fma(ve, W.ei[b][u], a[1]);
                        a[2] = fma(vo, W.qr[b][u], a[2]);
                        a[3] = fma(vo, W.qi[b][u], a[3]);
                    }
                }
                return;
            }
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                double *a = v + (s * NB + b) * 4;
                a[0] = u ? fma(ve, W.er[b][u], a[0]) : ve * W.er[b][u];
                a[1] = u ? fma(ve, W.ei[b][u], a[1]) : ve * W.ei[b][u];
                a[2] = u ? fma(vo, W.qr[b][u], a[2]) : vo * W.qr[b][u];
                a[3] = u ? fma(vo, W.qi[b][u], a[3]) : vo * W.qi[b][u];
            }
        });
    }
    const double s = warp_sums<TL * NB * 4>(v, lane);
    if (TL * NB * 4 == 32)
        red[lane] += s;
    else if (!(lane & 1))
        red[lane >> 1] += s;
}

// a block's steps [0, nk) (nk a multiple of TL; past lmax the coefficients are zero); groups that
// are evanescent as a whole run the recursion alone
template <int ZONE, int U, int NB, int TL>
__device__ __forceinline__ void anal_block(State<U> &S, const Weights<NB, U> &W, int nk, int &mode, const double2 *cf, double *red,
                                           int lane) {
    int k = 0;
    while (mode != CLEAN && k < nk) {
        if (mode == DEAD) {
#pragma unroll
            for (int s = 0; s < TL; ++s) two_step<ZONE>(S, cf[k + s], [](int, double, double) {});
        } else {
            anal_chunk<ZONE, true, U, NB, TL>(S, W, cf + k, red + k * NB * 4, lane);
        }
        k += TL;
        if (rescale(S, [](int) {})) mode = mode_of(S);
    }
#pragma unroll 1
    for (; k < nk; k += TL) anal_chunk<ZONE, false, U, NB, TL>(S, W, cf + k, red + k * NB * 4, lane);
}

// One CTA per (order, chunk of ring pairs or all of them in turn, NB maps), every warp keeping one group of
// 32 U pairs in registers over all l.  Per block of 256 l the warps' rows are summed by zone and combined to
//     a_l = N_k eps_{l+1} c_k + N_{k-1} eps_l c_{k-1} + M_l e_k,   a_{l+1} = N_k o_k + M_{l+1} o'_k.
template <int U, int NB, int TL, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) leg_analysis64_kernel(GeomDev g, LegTab tb, int lmax, int mmax,
                                                                  const double2 *__restrict__ Fm, int64_t fm_stride,
                                                                  double2 *__restrict__ alm, int64_t alm_stride, int nchunks,
                                                                  const int32_t *__restrict__ mlist) {
    constexpr int NW = NT / 32, ROW = LKB * NB * 4;
    __shared__ double2 ca[LKB], cb[LKB];
    __shared__ double cprev[2 * NB];
    __shared__ int wzone[NW];
    extern __shared__ double red[];  // [NW][LKB][NB][4], then the sums [zone][LKB][NB][4]
    double *sum = red + NW * ROW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // F row blockIdx.x holds order m (all orders, or the orders of mlist in list order)
    const int m = mlist ? mlist[blockIdx.x] : blockIdx.x;
    if (m < 0 || m > mmax) return;  // a listed order outside the plan: nothing read or written
    const int64_t np = g.npairs;
    const double2 *F = Fm + (int64_t)blockIdx.z * NB * fm_stride + (int64_t)blockIdx.x * np * 2;
    double *mine = red + warp * ROW;
    const bool atomic = gridDim.y > 1;
    for (int chunk = blockIdx.y; chunk < nchunks; chunk += gridDim.y) {
        const int grp = chunk * NW + warp;
        const double *tab = tb.row(m, 0);
        const bool any = (int64_t)grp * U * 32 < np;
        State<U> S;
        Weights<NB, U> W;
        const int zone = start_group(g, tab, m, grp, lane, S);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t p = unit_pair<U>(grp, u, lane);
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                W.er[b][u] = W.ei[b][u] = W.qr[b][u] = W.qi[b][u] = 0.0;
                if (p < np) {
                    const double2 fn = F[b * fm_stride + 2 * p], fs = F[b * fm_stride + 2 * p + 1];
                    const double x = zone == ZPOLE ? g.pair_x[p] : 1.0;
                    W.er[b][u] = fn.x + fs.x;
                    W.ei[b][u] = fn.y + fs.y;
                    W.qr[b][u] = (fn.x - fs.x) * x;
                    W.qi[b][u] = (fn.y - fs.y) * x;
                }
            }
        }
        int mode = mode_of(S);
        if (lane == 0) wzone[warp] = any ? zone : -1;
        for (int l0 = m; l0 <= lmax; l0 += 2 * LKB, tab += LKB * LT_N) {
            const int nk = min(LKB, (lmax - l0) / 2 + 1), nkp = (nk + TL - 1) / TL * TL;
            for (int i = tid; i < LKB; i += NT) {
                const double4 z = make_double4(0.0, 0.0, 0.0, 0.0);
                const double4 a = i < nk ? four(tab + (int64_t)i * LT_N + LT_A) : z, b = i < nk ? four(tab + (int64_t)i * LT_N + LT_B0) : z;
                ca[i] = make_double2(a.x, a.y);
                cb[i] = make_double2(b.x, b.y);
            }
            for (int i = lane; i < ROW; i += 32) mine[i] = 0.0;
            __syncthreads();
            if (any) {
                if (zone == ZPOLE)
                    anal_block<ZPOLE, U, NB, TL>(S, W, nkp, mode, ca, mine, lane);
                else
                    anal_block<ZEQ, U, NB, TL>(S, W, nkp, mode, cb, mine, lane);
            }
            __syncthreads();
            for (int i = tid; i < 2 * nk * NB * 4; i += NT) {
                const int z = i >= nk * NB * 4, o = i - z * nk * NB * 4;
                double s = 0.0;
                for (int w = 0; w < NW; ++w)
                    if (wzone[w] == z) s += red[w * ROW + o];
                sum[z * ROW + o] = s;
            }
            __syncthreads();
            for (int i = tid; i < nk * NB; i += NT) {
                const int k = i % nk, b = i / nk, l = l0 + 2 * k;
                const double *A = sum + (k * NB + b) * 4, *B = A + ROW, *t = tab + (int64_t)k * LT_N;
                double2 q = make_double2(0.0, 0.0);
                if (l > m) {
                    const double *c = k > 0 ? A - NB * 4 : cprev + 2 * b;
                    q = make_double2(t[LT_Q - LT_N] * c[0], t[LT_Q - LT_N] * c[1]);
                }
                const double2 v0 = make_double2(t[LT_P] * A[0] + t[LT_M0] * B[0] + q.x, t[LT_P] * A[1] + t[LT_M0] * B[1] + q.y);
                const double2 v1 = make_double2(t[LT_NX] * A[2] + t[LT_M1] * B[2], t[LT_NX] * A[3] + t[LT_M1] * B[3]);
                double2 *dst = alm + ((int64_t)blockIdx.z * NB + b) * alm_stride + alm_idx(lmax, l, m);
                if (atomic) {
                    atomicAdd(&dst[0].x, v0.x);
                    atomicAdd(&dst[0].y, v0.y);
                    if (l < lmax) {
                        atomicAdd(&dst[1].x, v1.x);
                        atomicAdd(&dst[1].y, v1.y);
                    }
                } else {  // the chunks before this one were added by this thread
                    dst[0] = chunk ? cadd(dst[0], v0) : v0;
                    if (l < lmax) dst[1] = chunk ? cadd(dst[1], v1) : v1;
                }
            }
            __syncthreads();
            if (tid < 2 * NB) cprev[tid] = sum[((LKB - 1) * NB + tid / 2) * 4 + tid % 2];
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ synthesis
struct alignas(16) ACoef {  // factors of the even and the odd value
    double cr, ci, dr, di;
};
template <int NB, int U> struct Sums {
    double er[NB][U], ei[NB][U], qr[NB][U], qi[NB][U];
};

template <int ZONE, int U, int NB>
__device__ __forceinline__ void synth_step(State<U> &S, Sums<NB, U> &A, double2 c, const ACoef *ac) {
    ACoef a[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) a[b] = ac[b * LKB];
    two_step<ZONE>(S, c, [&](int u, double ve, double vo) {
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            A.er[b][u] = fma(ve, a[b].cr, A.er[b][u]);
            A.ei[b][u] = fma(ve, a[b].ci, A.ei[b][u]);
            A.qr[b][u] = fma(vo, a[b].dr, A.qr[b][u]);
            A.qi[b][u] = fma(vo, a[b].di, A.qi[b][u]);
        }
    });
}

// the sums are kept in units of 2^(512 e); groups that are evanescent as a whole (below 2^-256)
// run the recursion alone
template <int ZONE, int U, int NB>
__device__ __forceinline__ void synth_block(State<U> &S, Sums<NB, U> &A, int nk, int &mode, const double2 *cf, const ACoef *ac) {
    int k = 0;
    while (mode != CLEAN && k < nk) {
        if (mode == DEAD) {
#pragma unroll
            for (int s = 0; s < 4; ++s) two_step<ZONE>(S, cf[k + s], [](int, double, double) {});
        } else {
#pragma unroll
            for (int s = 0; s < 4; ++s) synth_step<ZONE>(S, A, cf[k + s], ac + k + s);
        }
        k += 4;
        const bool up = rescale(S, [&](int u) {
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                A.er[b][u] *= 0x1p-512;
                A.ei[b][u] *= 0x1p-512;
                A.qr[b][u] *= 0x1p-512;
                A.qi[b][u] *= 0x1p-512;
            }
        });
        if (up) mode = mode_of(S);
    }
#pragma unroll 4
    for (; k < nk; ++k) synth_step<ZONE>(S, A, cf[k], ac + k);
}

// One warp per (group of 32 U ring pairs, order, NB maps): the warps of larger CTAs would wait for
// each other at every block, since those near the pole spend less on it.
template <int U, int NB, int MINB>
__global__ void __launch_bounds__(32, MINB) leg_synthesis64_kernel(GeomDev g, LegTab tb, int lmax, int mmax,
                                                                  const double2 *__restrict__ alm, int64_t alm_stride,
                                                                  double2 *__restrict__ Gm, int64_t gm_stride,
                                                                  const int32_t *__restrict__ mlist) {
    __shared__ double2 cf[LKB];
    __shared__ ACoef ac[NB * LKB];
    const int lane = threadIdx.x, grp = blockIdx.x;
    // G row blockIdx.y holds order m (all orders, or the orders of mlist in list order)
    const int m = mlist ? mlist[blockIdx.y] : blockIdx.y;
    if (m < 0 || m > mmax) return;  // a listed order outside the plan: nothing read or written
    const int64_t np = g.npairs;
    const double2 *a = alm + (int64_t)blockIdx.z * NB * alm_stride;
    const double *tab = tb.row(m, 0);
    State<U> S;
    Sums<NB, U> A;
    const int zone = start_group(g, tab, m, grp, lane, S);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int b = 0; b < NB; ++b) A.er[b][u] = A.ei[b][u] = A.qr[b][u] = A.qi[b][u] = 0.0;
    int mode = mode_of(S);
    for (int l0 = m; l0 <= lmax; l0 += 2 * LKB, tab += LKB * LT_N) {
        const int nk = min(LKB, (lmax - l0) / 2 + 1), nkp = (nk + 3) / 4 * 4;
        __syncwarp();
#pragma unroll
        for (int k = lane; k < LKB; k += 32) {
            const int l = l0 + 2 * k;
            double2 c = make_double2(0.0, 0.0);
            ACoef v[NB] = {};
            if (k < nk) {
                const double *t = tab + (int64_t)k * LT_N;
                const double4 f = four(t + (zone == ZPOLE ? LT_A : LT_B0));
                const double n = t[LT_NX];
                c = make_double2(f.x, f.y);
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const double2 *al = a + b * alm_stride + alm_idx(lmax, l, m);
                    const double2 z = make_double2(0.0, 0.0), a0 = al[0], a1 = l + 1 <= lmax ? al[1] : z;
                    if (zone == ZPOLE) {
                        const double2 a2 = l + 2 <= lmax ? al[2] : z;
                        v[b] = {f.z * a0.x + f.w * a2.x, f.z * a0.y + f.w * a2.y, n * a1.x, n * a1.y};
                    } else {
                        v[b] = {f.z * a0.x, f.z * a0.y, f.w * a1.x, f.w * a1.y};
                    }
                }
            }
            cf[k] = c;
#pragma unroll
            for (int b = 0; b < NB; ++b) ac[b * LKB + k] = v[b];
        }
        __syncwarp();
        if (zone == ZPOLE)
            synth_block<ZPOLE, U, NB>(S, A, nkp, mode, cf, ac);
        else
            synth_block<ZEQ, U, NB>(S, A, nkp, mode, cf, ac);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t p = unit_pair<U>(grp, u, lane);
        if (p >= np) continue;
        const double f = S.e[u] == 0 ? 1.0 : ldexp(1.0, 512 * S.e[u]), fq = zone == ZPOLE ? f * g.pair_x[p] : f;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            double2 *G = Gm + ((int64_t)blockIdx.z * NB + b) * gm_stride + ((int64_t)blockIdx.y * np + p) * 2;
            G[0] = make_double2(f * A.er[b][u] + fq * A.qr[b][u], f * A.ei[b][u] + fq * A.qi[b][u]);
            G[1] = make_double2(f * A.er[b][u] - fq * A.qr[b][u], f * A.ei[b][u] - fq * A.qi[b][u]);
        }
    }
}

// ------------------------------------------------------------------ launches
struct LegArgs {
    const hb_plan *p;
    int rows;
    const int32_t *mlist;
    cudaStream_t st;
    int64_t np() const { return p->g->d.npairs; }
    int64_t f_stride() const { return (int64_t)rows * np() * 2; }
    int64_t a_stride() const { return alm_size(p->lmax, p->mmax); }
};

template <int U, int NB, int TL, int NT, int MINB, bool IN_TURN>
static int run_analysis(const LegArgs &L, int nz, const double2 *F, double2 *alm) {
    const int64_t per = (int64_t)U * NT;
    const int nchunks = (int)((L.np() + per - 1) / per), ny = IN_TURN ? 1 : nchunks;
    if (ny > 1) HB_CUDA_TRY(cudaMemsetAsync(alm, 0, sizeof(double2) * L.a_stride() * NB * nz, L.st));
    const int smem = (NT / 32 + 2) * LKB * NB * 4 * (int)sizeof(double);
    const auto kernel = leg_analysis64_kernel<U, NB, TL, NT, MINB>;
    HB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    dim3 grid((unsigned)L.rows, (unsigned)ny, (unsigned)nz);
    kernel<<<grid, NT, smem, L.st>>>(L.p->g->d, L.p->leg, L.p->lmax, L.p->mmax, F, L.f_stride(), alm, L.a_stride(), nchunks,
                                     L.mlist);
    HB_CHECK_LAUNCH();
    return HB_OK;
}
template <int U, int NB, int MINB> static int run_synthesis(const LegArgs &L, int nz, const double2 *alm, double2 *G) {
    dim3 grid((unsigned)((L.np() + 32 * U - 1) / (32 * U)), (unsigned)L.rows, (unsigned)nz);
    leg_synthesis64_kernel<U, NB, MINB><<<grid, 32, 0, L.st>>>(L.p->g->d, L.p->leg, L.p->lmax, L.p->mmax, alm, L.a_stride(), G,
                                                               L.f_stride(), L.mlist);
    HB_CHECK_LAUNCH();
    return HB_OK;
}

// Pairs per lane and warps per CTA: large grids amortise the warp reduction (analysis) and the
// coefficient loads (synthesis) over U = 4 pairs per lane; grids below 1024 pairs spread their few
// pairs over more warps, since they do not fill the GPU.
// Analysis of large grids: every block of 256 l ends in a barrier of the CTA, where warps whose pairs are
// still evanescent wait for the others.  With IN_TURN a CTA has 4 warps and takes the chunks of an order
// one after the other (a fixed sum, no atomics), and the 3 or 4 CTAs of an SM fill each other's waits.  That
// takes enough orders (in_turn) and each of them once, which a list of orders does not promise; else one
// map's pairs run side by side, 16 warps a CTA.  In us, wide / in turn: nside 1024, one map, lmax 2047
// 1812 / 1680, 1100 553 / 534, 1000 456 / 459, 900 366 / 394.  Two maps, one by one wide / in pairs in turn: lmax 2047
// 3613 / 3015, 700 468 / 415, 500 242 / 277 (in pairs wide, 8 warps: 4302, 560, 289).
static bool in_turn(const LegArgs &L, int nb, int64_t nz) {
    return L.np() >= 1024 && !L.mlist && L.rows * nz >= (nb == 1 ? 1024 : 512);
}
template <int NB> static int analysis_nb(const LegArgs &L, int nz, const double2 *F, double2 *alm) {
    constexpr int TL = NB == 1 ? 4 : 2;
    if ((NB == 2 && L.np() >= 1024) || in_turn(L, NB, nz)) return run_analysis<4, NB, TL, 128, NB == 1 ? 4 : 3, true>(L, nz, F, alm);
    if (NB == 1 && L.np() >= 1024) return run_analysis<4, 1, 4, 512, 0, false>(L, nz, F, alm);
    if (L.np() >= 256) return run_analysis<2, NB, TL, 256, 0, false>(L, nz, F, alm);
    return run_analysis<1, NB, TL, 128, 0, false>(L, nz, F, alm);
}
template <int NB> static int synthesis_nb(const LegArgs &L, int nz, const double2 *alm, double2 *G) {
    if (L.np() >= 1024) return run_synthesis<NB == 1 ? 4 : 2, NB, NB == 1 ? 16 : 14>(L, nz, alm, G);
    return run_synthesis<1, NB, 16>(L, nz, alm, G);
}

// Maps in pairs that share one recursion: 11 operations per (two l, ring pair) for two maps, 7 for one.
// Below 256 ring pairs one launch of single maps: these are bound by latency (3 maps at nside 64, lmax 100:
// 6 us, 9 us as a pair and a single).
template <typename Fn2, typename Fn1> static int by_two(int nmaps, bool pairs, Fn2 f2, Fn1 f1) {
    const int n2 = pairs ? nmaps / 2 : 0;
    if (n2)
        if (int rc = f2(n2, 0)) return rc;
    return nmaps > 2 * n2 ? f1(nmaps - 2 * n2, 2 * n2) : HB_OK;
}

int launch_leg_analysis64(const hb_plan *p, int nmaps, const double2 *F, double2 *alm, cudaStream_t st, int nm,
                          const int32_t *mlist) {
    const LegArgs L{p, mlist ? nm : p->mmax + 1, mlist, st};
    const int64_t fs = L.f_stride(), as = L.a_stride();
    const bool pairs = L.np() >= 1024 ? in_turn(L, 2, nmaps / 2) : L.np() >= 256;
    return by_two(nmaps, pairs, [&](int nz, int b) { return analysis_nb<2>(L, nz, F + b * fs, alm + b * as); },
                  [&](int nz, int b) { return analysis_nb<1>(L, nz, F + b * fs, alm + b * as); });
}

int launch_leg_synthesis64(const hb_plan *p, int nmaps, const double2 *alm, double2 *G, cudaStream_t st, int nm,
                           const int32_t *mlist) {
    const LegArgs L{p, mlist ? nm : p->mmax + 1, mlist, st};
    const int64_t fs = L.f_stride(), as = L.a_stride();
    return by_two(nmaps, L.np() >= 256, [&](int nz, int b) { return synthesis_nb<2>(L, nz, alm + b * as, G + b * fs); },
                  [&](int nz, int b) { return synthesis_nb<1>(L, nz, alm + b * as, G + b * fs); });
}

}  // namespace hb
