// Spin-2 (Q/U <-> E/B) Legendre kernels in FP64 (the FP32 ones are in hb_spin32.cu), and the launchers
// of both.
//
// Replaces map2alm_spin_gpu / eb_from_qu_gpu / qu_from_eb_gpu (spin.py:32-115) and the
// closed-form Wigner sum wigner_d_ms_sum (wigner_d_ms.cu:20-50, one launch per (m, s), O(lmax^2)
// per ring, overflowing lgamma/exp terms).  Convention (HEALPix / Zaldarriaga-Seljak, one
// consistent choice; the reference's inverse uses a2 = -(E - iB) (spin.py:84), which contradicts
// its forward):
//     _sY_lm = _s lambda_lm(theta) e^{i m phi},   _s lambda_lm = sqrt((2l+1)/4pi) d^l_{m,-s}(theta)
//     E = -(a2 + a-2)/2,  B = i (a2 - a-2)/2,  a(+-2) = -(E +- i B).
// P = _{+2}lambda and M = _{-2}lambda on the north ring of a pair come from the three-term
// Wigner recursion in l (same a_l, c_l; opposite sign of the m*s term):
//     P_{l+1} = (a_l x + b_l) P_l - c_l P_{l-1},   M_{l+1} = (a_l x - b_l) M_l - c_l M_{l-1},
//     a_l = (N_{l+1}/N_l)(2l+1)(l+1)/R_{l+1},  b_l = (N_{l+1}/N_l)(2l+1) 2m/(l R_{l+1}),
//     c_l = (N_{l+1}/N_{l-1})(l+1) R_l/(l R_{l+1}),  R_l = sqrt((l^2-m^2)(l^2-4)),
// started at l0 = max(m,2) from the closed-form d^{l0}_{m,+-2} (log-scaled; P and M carry
// separate running exponents: their ratio near the poles is cot^4(theta/2)).
// Mirror symmetry: _s lambda(pi - theta) = (-1)^(l+m) _{-s}lambda(theta).
//
// The recursions run scaled, P_l = N_l rho_l with N_l N_{l+1} eps_{l+1} = 1/2, eps_l = 1 / a_{l-1}:
//     rho_{l+1} = (A_l x +- A_l beta_l) rho_l - rho_{l-1},   A_l = 2 N_l^2,  beta_l = 2m / (l (l+1)),
// 2 operations per function and l instead of 5.  N_l follows from its products over l, scanned by a
// warp when a block's coefficients are staged.  Values are mantissa * 2^(512 e) and count as zero while
// e < 0 (below 2^-256).
//
// What bounds the kernels: the FP64 pipe, 4 operations per (l, ring pair) for the recursions and 8 per map
// for the contraction, and in the analysis the warp reductions.  Three Q/U maps at nside 256, lmax 700:
// synthesis 523 -> 440 us, analysis 1261 -> 593 us.
#include <cmath>

#include "hb_internal.cuh"
#include "hb_warp.cuh"

namespace hb {

constexpr int SPB = 128;  // l per staged block

// log-scaled start values of P (d_{m,-2}) and M (d_{m,+2}) at l0 = max(m, 2)
__device__ __forceinline__ void spin_start64(const GeomDev &g, int m, int64_t p, double &mp, int &ep, double &mm, int &em) {
    const double lc = g.pair_log2ch[p], ls = g.pair_log2sh[p], k = g.log2spin[m];
    const int u = m + 2, v = m >= 2 ? m - 2 : 2 - m;
    const double LP = k + v * lc + u * ls, LM = k + u * lc + v * ls;
    const double sp = (m & 1) ? -1.0 : 1.0, sm = (m >= 2) ? sp : 1.0;
    ep = (int)floor((LP + 256.0) / 512.0);
    em = (int)floor((LM + 256.0) / 512.0);
    mp = sp * exp2(LP - 512.0 * ep);
    mm = sm * exp2(LM - 512.0 * em);
}

// eps_l^2 = (l^2 - m^2)(l^2 - 4) / (l^2 (4 l^2 - 1))
__device__ __forceinline__ double spin_eps2(int l, int m) {
    const double ll = l, mm = m, l2 = ll * ll;
    return ((ll - mm) * (ll + mm) * (l2 - 4.0)) / (l2 * (4.0 * l2 - 1.0));
}
// A of the first l: the smooth choice (N = (2 eps)^-1/2), so that N stays of order one
__device__ __forceinline__ double spin_a0(int l0, int m) { return rsqrt(spin_eps2(l0 + 1, m)); }

// Step coefficients of rows l0 .. l0 + SPB - 1 by one warp: cf = (A, A beta) taking rho_l to rho_{l+1}, nl =
// N_l.  carry: A_{l0}, updated for the next block.  Even rows: A_{l+2} = A_l eps_{l+1}^2 / eps_{l+2}^2, each
// lane multiplying its two ratios, a scan over the lanes joining them.  Odd rows follow from the row
// before, A_l A_{l+1} eps_{l+1}^2 = 1, so that rounding cannot drift in that product (it acts like a change
// of x: two independent chains gave 20 to 100 times the error).
__device__ __forceinline__ void spin_rows(int l0, int m, int lane, double2 *cf, double *nl, double &carry) {
    const int l = l0 + 4 * lane;
    double e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = spin_eps2(l + 1 + i, m);
    const double q = e[0] / e[1];
    double pe = q * (e[2] / e[3]);  // A_{l+4} / A_l
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double a = __shfl_up_sync(0xffffffffu, pe, o);
        if (lane >= o) pe *= a;
    }
    double xe = __shfl_up_sync(0xffffffffu, pe, 1);
    if (lane == 0) xe = 1.0;
    double A[4];
    A[0] = carry * xe;
    A[1] = 1.0 / (e[0] * A[0]);
    A[2] = A[0] * q;
    A[3] = 1.0 / (e[2] * A[2]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double dl = (double)(l + i);
        cf[4 * lane + i] = make_double2(A[i], A[i] * (2.0 * m) / (dl * (dl + 1.0)));
        nl[4 * lane + i] = sqrt(0.5 * A[i]);
    }
    carry *= __shfl_sync(0xffffffffu, pe, 31);
}

enum { CLEAN = 0, MIXED = 1, DEAD = 2 };  // no / some / every value of the warp's group has e < 0

// U ring pairs per lane of one warp: pair 32 (grp U + u) + lane.  (p1, m1) at l, (p0, m0) at l - 1
template <int U> struct State {
    double p1[U], p0[U], m1[U], m0[U], x[U];
    int ep[U], em[U];
};

template <int U> __device__ __forceinline__ void start_group(const GeomDev &g, int m, int l0, int grp, int lane, State<U> &S) {
    const double inv = 1.0 / sqrt(0.5 * spin_a0(l0, m));  // 1 / N_{l0}
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t p = (int64_t)(grp * U + u) * 32 + lane;
        S.p1[u] = S.p0[u] = S.m1[u] = S.m0[u] = S.x[u] = 0.0;
        S.ep[u] = S.em[u] = 0;
        if (p < g.npairs) {
            S.x[u] = g.pair_x[p];
            spin_start64(g, m, p, S.p1[u], S.ep[u], S.m1[u], S.em[u]);
            S.p1[u] *= inv;
            S.m1[u] *= inv;
        }
    }
}

// hands (P_l, M_l) to f(u, P, M), then takes the step to l + 1
template <int U, typename Fn> __device__ __forceinline__ void spin_step(State<U> &S, double2 c, Fn f) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const double p = S.p1[u], q = S.m1[u];
        f(u, p, q);
        S.p1[u] = fma(fma(c.x, S.x[u], c.y), p, -S.p0[u]);
        S.m1[u] = fma(fma(c.x, S.x[u], -c.y), q, -S.m0[u]);
        S.p0[u] = p;
        S.m0[u] = q;
    }
}

template <int U> __device__ __forceinline__ int mode_of(const State<U> &S) {
    bool neg = false, live = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        neg |= (S.ep[u] < 0) | (S.em[u] < 0);
        live |= (S.ep[u] >= 0) | (S.em[u] >= 0);
    }
    if (!__any_sync(0xffffffffu, neg)) return CLEAN;
    return __any_sync(0xffffffffu, live) ? MIXED : DEAD;
}

__device__ __forceinline__ bool past(double v) { return (__double2hiint(v) & 0x7fffffff) >= 0x4ff00000; }  // |v| >= 2^256

// values that have grown past 2^256 move to the next exponent; upP(u), upM(u) are told.  False when the
// warp has none.
template <int U, typename FP, typename FM> __device__ __forceinline__ bool rescale(State<U> &S, FP upP, FM upM) {
    bool any = false;
#pragma unroll
    for (int u = 0; u < U; ++u) any |= (S.ep[u] < 0 && past(S.p1[u])) || (S.em[u] < 0 && past(S.m1[u]));
    if (!__any_sync(0xffffffffu, any)) return false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (S.ep[u] < 0 && past(S.p1[u])) {
            S.p1[u] *= 0x1p-512;
            S.p0[u] *= 0x1p-512;
            ++S.ep[u];
            upP(u);
        }
        if (S.em[u] < 0 && past(S.m1[u])) {
            S.m1[u] *= 0x1p-512;
            S.m0[u] *= 0x1p-512;
            ++S.em[u];
            upM(u);
        }
    }
    return true;
}

// ------------------------------------------------------------------ analysis
// With eps = (-1)^(l-m), Qe = QN + eps QS, Qo = QN - eps QS (U alike): E += P w + M v, B += -i P w' + i M v',
// w = -(Qe + i Uo)/2, v = -(Qe - i Uo)/2 and w', v' the same of the other parity.
template <int U> struct Weights {
    double2 w[2][U], v[2][U];  // [l - m even, odd]
};

// Four rows: sums over the group's pairs, added to the warp's row red[row * 4 + (E re, E im, B re, B im)].  GATED:
// P and M with e < 0 take no part, their terms predicated off (as in the scalar analysis; three maps at nside 256,
// lmax 700, whole call 734 us, 764 with zeroed values; one at nside 1024, lmax 2047 5882, 5957).
template <bool GATED, int U, int PAR>
__device__ __forceinline__ void anal_chunk(State<U> &S, const Weights<U> &W, const double2 *cf, double *red, int lane) {
    double a[16];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int k = (s + PAR) & 1;
        spin_step(S, cf[s], [&](int u, double p, double q) {
            const double2 w = W.w[k][u], v = W.v[k][u], wo = W.w[k ^ 1][u], vo = W.v[k ^ 1][u];
            double *o = a + 4 * s;
            if (GATED) {
                if (u == 0) o[0] = o[1] = o[2] = o[3] = 0.0;
                if (S.em[u] >= 0) {
                    o[0] = fma(q, v.x, o[0]);
                    o[1] = fma(q, v.y, o[1]);
                    o[2] = fma(-q, vo.y, o[2]);
                    o[3] = fma(q, vo.x, o[3]);
                }
                if (S.ep[u] >= 0) {
                    o[0] = fma(p, w.x, o[0]);
                    o[1] = fma(p, w.y, o[1]);
                    o[2] = fma(p, wo.y, o[2]);
                    o[3] = fma(-p, wo.x, o[3]);
                }
                return;
            }
            o[0] = fma(p, w.x, u ? fma(q, v.x, o[0]) : q * v.x);
            o[1] = fma(p, w.y, u ? fma(q, v.y, o[1]) : q * v.y);
            o[2] = fma(p, wo.y, u ? fma(-q, vo.y, o[2]) : -q * vo.y);
            o[3] = fma(-p, wo.x, u ? fma(q, vo.x, o[3]) : q * vo.x);
        });
    }
    const double t = warp_sums<16>(a, lane);
    if (!(lane & 1)) red[lane >> 1] += t;
}

template <int U, int PAR>
__device__ __forceinline__ void anal_block(State<U> &S, const Weights<U> &W, int n, int &mode, const double2 *cf, double *red, int lane) {
    int k = 0;
    while (mode != CLEAN && k < n) {
        if (mode == DEAD) {
#pragma unroll
            for (int s = 0; s < 4; ++s) spin_step(S, cf[k + s], [](int, double, double) {});
        } else {
            anal_chunk<true, U, PAR>(S, W, cf + k, red + 4 * k, lane);
        }
        k += 4;
        if (rescale(S, [](int) {}, [](int) {})) mode = mode_of(S);
    }
#pragma unroll 1
    for (; k < n; k += 4) anal_chunk<false, U, PAR>(S, W, cf + k, red + 4 * k, lane);
}

// One CTA per (order, chunk of ring pairs, map), every warp keeping one group of 32 U pairs in registers
// over all l
template <int U, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) spin_analysis64_kernel(GeomDev g, int lmax, const double2 *__restrict__ QF,
                                                                   const double2 *__restrict__ UF, int64_t fm_stride,
                                                                   double2 *__restrict__ Eo, double2 *__restrict__ Bo,
                                                                   int64_t alm_stride, int atomic) {
    constexpr int NW = NT / 32, ROW = SPB * 4;
    __shared__ double2 cf[SPB];
    __shared__ double nl[SPB];
    extern __shared__ double red[];  // [NW][SPB][4]
    const int m = blockIdx.x, b = blockIdx.z, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, grp = blockIdx.y * NW + warp;
    const int ls = m > 2 ? m : 2, par0 = (ls - m) & 1;
    const int64_t np = g.npairs;
    const double2 *Qf = QF + b * fm_stride + (int64_t)m * np * 2, *Uf = UF + b * fm_stride + (int64_t)m * np * 2;
    double2 *E = Eo + b * alm_stride, *B = Bo + b * alm_stride;
    if (!atomic && tid < 2 && m + tid < ls && m + tid <= lmax)  // E, B are zero for l < 2
        E[alm_idx(lmax, m + tid, m)] = B[alm_idx(lmax, m + tid, m)] = make_double2(0.0, 0.0);
    if (ls > lmax) return;
    State<U> S;
    Weights<U> W;
    start_group(g, m, ls, grp, lane, S);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t p = (int64_t)(grp * U + u) * 32 + lane;
        double2 qn = make_double2(0.0, 0.0), qs = qn, un = qn, us = qn;
        if (p < np) {
            qn = Qf[2 * p];
            qs = Qf[2 * p + 1];
            un = Uf[2 * p];
            us = Uf[2 * p + 1];
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const double2 Qe = k ? csub(qn, qs) : cadd(qn, qs), Uo = k ? cadd(un, us) : csub(un, us);
            W.w[k][u] = make_double2(-0.5 * (Qe.x - Uo.y), -0.5 * (Qe.y + Uo.x));
            W.v[k][u] = make_double2(-0.5 * (Qe.x + Uo.y), -0.5 * (Qe.y - Uo.x));
        }
    }
    const bool any = (int64_t)grp * U * 32 < np;
    int mode = mode_of(S);
    double *mine = red + warp * ROW;
    double carry = spin_a0(ls, m);
    for (int l0 = ls; l0 <= lmax; l0 += SPB) {
        const int n = min(SPB, lmax - l0 + 1), npd = (n + 3) & ~3;
        if (warp == 0) spin_rows(l0, m, lane, cf, nl, carry);
        for (int i = lane; i < ROW; i += 32) mine[i] = 0.0;
        __syncthreads();
        if (any) {
            if (par0)
                anal_block<U, 1>(S, W, npd, mode, cf, mine, lane);
            else
                anal_block<U, 0>(S, W, npd, mode, cf, mine, lane);
        }
        __syncthreads();
        for (int i = tid; i < 2 * n; i += NT) {
            const int row = i >> 1, c = (i & 1) * 2;  // E or B of the row
            double2 s = make_double2(0.0, 0.0);
            for (int w = 0; w < NW; ++w) {
                s.x += red[w * ROW + 4 * row + c];
                s.y += red[w * ROW + 4 * row + c + 1];
            }
            s = cscale(s, nl[row]);
            double2 *d = (c ? B : E) + alm_idx(lmax, l0 + row, m);
            if (atomic) {
                atomicAdd(&d->x, s.x);
                atomicAdd(&d->y, s.y);
            } else {
                *d = s;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ synthesis
// With A+ = E + iB, A- = E - iB and eps = (-1)^(l-m):
//   north: Q = -1/2 sum (P A+ + M A-),      U = -i/2 sum (M A- - P A+),
//   south: Q = -1/2 sum eps (P A- + M A+),  U = -i/2 sum eps (P A- - M A+).
// The sums of P and M stay apart (their exponents differ), in units of 2^(512 e).
template <int U> struct Sums {
    double2 x1[U], x2[U], x3[U], x4[U];  // P A+, M A-, eps P A-, eps M A+
};
struct alignas(16) SAlm {
    double pr, pi, mr, mi;  // N (A+, A-)
};
__device__ __forceinline__ void axpy(double2 &s, double v, double r, double i) {
    s.x = fma(v, r, s.x);
    s.y = fma(v, i, s.y);
}

template <int U>
__device__ __forceinline__ void synth_row(State<U> &S, Sums<U> &A, double2 c, const SAlm &a, bool odd) {
    spin_step(S, c, [&](int u, double p, double q) {
        axpy(A.x1[u], p, a.pr, a.pi);
        axpy(A.x2[u], q, a.mr, a.mi);
        axpy(A.x3[u], odd ? -p : p, a.mr, a.mi);
        axpy(A.x4[u], odd ? -q : q, a.pr, a.pi);
    });
}

template <int U, int PAR>
__device__ __forceinline__ void synth_block(State<U> &S, Sums<U> &A, int n, int &mode, const double2 *cf, const SAlm *ac) {
    int k = 0;
    while (mode != CLEAN && k < n) {
        if (mode == DEAD) {
#pragma unroll
            for (int s = 0; s < 4; ++s) spin_step(S, cf[k + s], [](int, double, double) {});
        } else {
#pragma unroll
            for (int s = 0; s < 4; ++s) synth_row(S, A, cf[k + s], ac[k + s], (s + PAR) & 1);
        }
        k += 4;
        const auto down = [](double2 &v) { v = cscale(v, 0x1p-512); };
        const bool up = rescale(
            S,
            [&](int u) {
                down(A.x1[u]);
                down(A.x3[u]);
            },
            [&](int u) {
                down(A.x2[u]);
                down(A.x4[u]);
            });
        if (up) mode = mode_of(S);
    }
#pragma unroll 1
    for (; k < n; k += 4) {
#pragma unroll
        for (int s = 0; s < 4; ++s) synth_row(S, A, cf[k + s], ac[k + s], (s + PAR) & 1);
    }
}

// One warp per (group of 32 U ring pairs, order, map), as in the scalar synthesis
template <int U, int MINB>
__global__ void __launch_bounds__(32, MINB) spin_synthesis64_kernel(GeomDev g, int lmax, const double2 *__restrict__ E,
                                                                   const double2 *__restrict__ B, int64_t alm_stride,
                                                                   double2 *__restrict__ QG, double2 *__restrict__ UG,
                                                                   int64_t gm_stride) {
    __shared__ double2 cf[SPB];
    __shared__ double nl[SPB];
    __shared__ SAlm ac[SPB];
    const int lane = threadIdx.x, grp = blockIdx.x, m = blockIdx.y;
    const int ls = m > 2 ? m : 2, par0 = (ls - m) & 1;
    const int64_t np = g.npairs;
    const double2 *Eb = E + blockIdx.z * alm_stride, *Bb = B + blockIdx.z * alm_stride;
    State<U> S;
    Sums<U> A;
    start_group(g, m, ls, grp, lane, S);
#pragma unroll
    for (int u = 0; u < U; ++u) A.x1[u] = A.x2[u] = A.x3[u] = A.x4[u] = make_double2(0.0, 0.0);
    int mode = mode_of(S);
    double carry = spin_a0(ls, m);
    for (int l0 = ls; l0 <= lmax; l0 += SPB) {
        const int n = min(SPB, lmax - l0 + 1), npd = (n + 3) & ~3;
        __syncwarp();
        spin_rows(l0, m, lane, cf, nl, carry);
        __syncwarp();
#pragma unroll
        for (int k = lane; k < SPB; k += 32) {
            SAlm v{};
            if (k < n) {
                const double2 e = Eb[alm_idx(lmax, l0 + k, m)], bv = Bb[alm_idx(lmax, l0 + k, m)];
                const double N = nl[k];
                v = {N * (e.x - bv.y), N * (e.y + bv.x), N * (e.x + bv.y), N * (e.y - bv.x)};
            }
            ac[k] = v;
        }
        __syncwarp();
        if (par0)
            synth_block<U, 1>(S, A, npd, mode, cf, ac);
        else
            synth_block<U, 0>(S, A, npd, mode, cf, ac);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t p = (int64_t)(grp * U + u) * 32 + lane;
        if (p >= np) continue;
        const double fp = S.ep[u] == 0 ? 1.0 : ldexp(1.0, 512 * S.ep[u]), fm = S.em[u] == 0 ? 1.0 : ldexp(1.0, 512 * S.em[u]);
        const double2 x1 = cscale(A.x1[u], fp), x3 = cscale(A.x3[u], fp), x2 = cscale(A.x2[u], fm), x4 = cscale(A.x4[u], fm);
        const double2 dn = csub(x2, x1), ds = csub(x3, x4);
        const int64_t o = blockIdx.z * gm_stride + ((int64_t)m * np + p) * 2;
        QG[o] = cscale(cadd(x1, x2), -0.5);
        QG[o + 1] = cscale(cadd(x3, x4), -0.5);
        UG[o] = make_double2(0.5 * dn.y, -0.5 * dn.x);  // -i/2 z
        UG[o + 1] = make_double2(0.5 * ds.y, -0.5 * ds.x);
    }
}

// ------------------------------------------------------------------ launches
template <int U, int NT, int MINB>
static int run_analysis(const hb_plan *p, int nmaps, const double2 *QF, const double2 *UF, double2 *E, double2 *B, cudaStream_t st) {
    const int64_t np = p->g->d.npairs, as = alm_size(p->lmax, p->mmax), per = (int64_t)U * NT;
    const int nchunks = (int)((np + per - 1) / per);
    if (nchunks > 1) {
        HB_CUDA_TRY(cudaMemsetAsync(E, 0, sizeof(double2) * as * nmaps, st));
        HB_CUDA_TRY(cudaMemsetAsync(B, 0, sizeof(double2) * as * nmaps, st));
    }
    const int smem = NT / 32 * SPB * 4 * (int)sizeof(double);
    HB_CUDA_TRY(cudaFuncSetAttribute(spin_analysis64_kernel<U, NT, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    dim3 grid((unsigned)(p->mmax + 1), (unsigned)nchunks, (unsigned)nmaps);
    spin_analysis64_kernel<U, NT, MINB><<<grid, NT, smem, st>>>(p->g->d, p->lmax, QF, UF, (int64_t)(p->mmax + 1) * np * 2, E, B, as,
                                                                nchunks > 1);
    HB_CHECK_LAUNCH();
    return HB_OK;
}
template <int U, int MINB>
static int run_synthesis(const hb_plan *p, int nmaps, const double2 *E, const double2 *B, double2 *QG, double2 *UG, cudaStream_t st) {
    const int64_t np = p->g->d.npairs;
    dim3 grid((unsigned)((np + 32 * U - 1) / (32 * U)), (unsigned)(p->mmax + 1), (unsigned)nmaps);
    spin_synthesis64_kernel<U, MINB><<<grid, 32, 0, st>>>(p->g->d, p->lmax, E, B, alm_size(p->lmax, p->mmax), QG, UG,
                                                              (int64_t)(p->mmax + 1) * np * 2);
    HB_CHECK_LAUNCH();
    return HB_OK;
}

// Pairs per lane: the synthesis reads 48 bytes of coefficients per l and warp from shared memory, as long
// as the operations of two pairs; four pairs (10 warps per SM) 3.88 ms at nside 1024 where two (16 warps)
// take 4.09, but 464 us at nside 256, lmax 700 (three maps) where two take 439.  The analysis: four 5.25 ms
// and 593 us, two (with the gate on the values) 6.06 ms and 667 us.  Below 256 pairs one, to spread over more warps.
static int spin_analysis64(const hb_plan *p, int nmaps, const double2 *QF, const double2 *UF, double2 *E, double2 *B, cudaStream_t st) {
    if (p->g->d.npairs >= 256) return run_analysis<4, 128, 3>(p, nmaps, QF, UF, E, B, st);
    return run_analysis<1, 128, 4>(p, nmaps, QF, UF, E, B, st);
}
static int spin_synthesis64(const hb_plan *p, int nmaps, const double2 *E, const double2 *B, double2 *QG, double2 *UG, cudaStream_t st) {
    if (p->g->d.npairs >= 1024) return run_synthesis<4, 10>(p, nmaps, E, B, QG, UG, st);
    if (p->g->d.npairs >= 256) return run_synthesis<2, 16>(p, nmaps, E, B, QG, UG, st);
    return run_synthesis<1, 16>(p, nmaps, E, B, QG, UG, st);
}

int launch_spin_analysis32(const hb_plan *p, int nmaps, const float2 *QF, const float2 *UF, float2 *E, float2 *B, cudaStream_t st);
int launch_spin_synthesis32(const hb_plan *p, int nmaps, const float2 *E, const float2 *B, float2 *QG, float2 *UG, cudaStream_t st);

int launch_spin_analysis(const hb_plan *p, int precision, int nmaps, const void *QFm, const void *UFm, void *E, void *B,
                         cudaStream_t st) {
    HB_NVTX("spin_analysis");
    if (precision == 32)
        return launch_spin_analysis32(p, nmaps, (const float2 *)QFm, (const float2 *)UFm, (float2 *)E, (float2 *)B, st);
    return spin_analysis64(p, nmaps, (const double2 *)QFm, (const double2 *)UFm, (double2 *)E, (double2 *)B, st);
}

int launch_spin_synthesis(const hb_plan *p, int precision, int nmaps, const void *E, const void *B, void *QGm, void *UGm,
                          cudaStream_t st) {
    HB_NVTX("spin_synthesis");
    if (precision == 32)
        return launch_spin_synthesis32(p, nmaps, (const float2 *)E, (const float2 *)B, (float2 *)QGm, (float2 *)UGm, st);
    return spin_synthesis64(p, nmaps, (const double2 *)E, (const double2 *)B, (double2 *)QGm, (double2 *)UGm, st);
}

}  // namespace hb
