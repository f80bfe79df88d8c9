// Spin-2 (Q/U <-> E/B) Legendre kernels in FP32 (conventions and recursion: hb_spin.cu, which holds the
// FP64 ones).
//
// P = _{+2}lambda and M = _{-2}lambda of a ring pair's north ring run side by side,
//     P_l = a (x P_{l-1}) + b P_{l-1} - c P_{l-2},   M_l = a (x M_{l-1}) - b M_{l-1} - c M_{l-2},
// with x as a float pair, restarting every 256 l from the plan's FP64-computed checkpoints; states
// are mantissa * 2^(64 e) with separate exponents, moved to the next one after every fourth l.
//
// What bounds the kernels: the FMA pipe, 10 operations per (l, ring pair) for the recursions and 8 for
// the contraction.  All of them are packed (fma.rn.f32x2), which leaves half the issue slots to loads
// and to the analysis's reduction; pairs that stay evanescent over a block of 256 l are skipped by
// the plan's flags, and the coefficients are a table of the plan.
// One Q/U map at nside 1024, lmax 2047: synthesis 3850 -> 2360 us, analysis 6120 -> 3660 us (scalar
// instructions before, 16 weights reloaded from global memory, no skip); the analysis gives the same bits.
#include <cmath>

#include "hb_f32x2.cuh"
#include "hb_internal.cuh"

namespace hb {

constexpr int SB = 256;  // l per block (the checkpoint spacing)

// log-scaled start values of P (d_{m,-2}) and M (d_{m,+2}) at l0 = max(m, 2)
__device__ __forceinline__ void spin_start32(const GeomDev &g, int m, int64_t p, float &mp, int &ep, float &mm, int &em) {
    const double lc = g.pair_log2ch[p], ls = g.pair_log2sh[p], k = g.log2spin[m];
    const int u = m + 2, v = m >= 2 ? m - 2 : 2 - m;
    const double LP = k + v * lc + u * ls, LM = k + u * lc + v * ls;
    const double sp = (m & 1) ? -1.0 : 1.0, sm = (m >= 2) ? sp : 1.0;
    ep = (int)floor((LP + 32.0) / 64.0);
    em = (int)floor((LM + 32.0) / 64.0);
    mp = (float)(sp * exp2(LP - 64.0 * ep));
    mm = (float)(sm * exp2(LM - 64.0 * em));
}

struct SpinPair {  // (P, M) values of l - 1 and l - 2 and their exponents at a block's start
    float p1, p2, m1, m2;
    int ep, em;
};
__device__ __forceinline__ SpinPair spin_state(const GeomDev &g, int m, int j, int64_t p, const float4 *ckP, const float4 *ckM) {
    SpinPair s{};
    if (p >= g.npairs) return s;
    if (j == 0) {
        spin_start32(g, m, p, s.p2, s.ep, s.m2, s.em);
    } else {
        const float4 cp = ckP[p], cm = ckM[p];
        s.p1 = cp.x;
        s.p2 = cp.y;
        s.ep = __float_as_int(cp.z);
        s.m1 = cm.x;
        s.m2 = cm.y;
        s.em = __float_as_int(cm.z);
    }
    return s;
}

// one recursion step: a xm(v1) + (b v1 - c v2), nc = -c
__device__ __forceinline__ f32x2 spin_step(f32x2 a, f32x2 b, f32x2 nc, f32x2 xh, f32x2 xl, f32x2 v1, f32x2 v2) {
    return fma2(a, fma2(xh, v1, mul2(xl, v1)), fma2(b, v1, mul2(nc, v2)));
}

// ------------------------------------------------------------------ analysis
// One CTA per (block of 256 l, order, map), the chunks of K NT ring pairs one after the other, no atomics.
// The sum over a chunk runs in a fixed order: thread t adds its K pairs k NT + t (M before P), columns
// t = s + SUBS j add up over j = 0 .. 15 through shared memory (RB rows at a time, double buffered), and
// the SUBS = NT / 16 results form a binary tree.  The recursions are packed over a thread's pairs, the
// contraction over (re, im).
//
// Weights per pair and slot parity q (l - m parity q ^ par0):  E += P wpe + M wme,  B += P wpb + M wmb
// with eps = (-1)^(l-m), Qe = QN + eps QS, Qo = QN - eps QS (U alike):
//   wpe = -(Qe + i Uo)/2, wme = -(Qe - i Uo)/2, wpb = -(Ue - i Qo)/2, wmb = -(Ue + i Qo)/2.
template <int K> struct SpinW {
    f32x2 pe[2][K], me[2][K], pb[2][K], mb[2][K];
};

template <int K>
__device__ __forceinline__ void spin_weights(SpinW<K> &W, int k, float4 Q, float4 U, int par0, bool gp, bool gm) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float eps = ((q ^ par0) & 1) ? -1.f : 1.f, h = -0.5f;
        const float2 Qe = make_float2(Q.x + eps * Q.z, Q.y + eps * Q.w), Qo = make_float2(Q.x - eps * Q.z, Q.y - eps * Q.w);
        const float2 Ue = make_float2(U.x + eps * U.z, U.y + eps * U.w), Uo = make_float2(U.x - eps * U.z, U.y - eps * U.w);
        W.pe[q][k] = gp ? pk(h * (Qe.x - Uo.y), h * (Qe.y + Uo.x)) : 0;
        W.me[q][k] = gm ? pk(h * (Qe.x + Uo.y), h * (Qe.y - Uo.x)) : 0;
        W.pb[q][k] = gp ? pk(h * (Ue.x + Qo.y), h * (Ue.y - Qo.x)) : 0;
        W.mb[q][k] = gm ? pk(h * (Ue.x - Qo.y), h * (Ue.y + Qo.x)) : 0;
    }
}

struct alignas(16) SpinCoefA {  // (a, a), (b, b), (-b, -b), (-c, -c)
    f32x2 a, b, nb, nc;
};

// K: pairs per thread, KS: of the sum's order (1 when K = 2 stands for it)
template <int KS, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) spin_analysis32_kernel(GeomDev g, int lmax, int mmax, const float2 *__restrict__ QF,
                                                                   const float2 *__restrict__ UF, int64_t fm_stride,
                                                                   float2 *__restrict__ Eo, float2 *__restrict__ Bo,
                                                                   int64_t alm_stride, const float4 *__restrict__ ckP,
                                                                   const float4 *__restrict__ ckM,
                                                                   const uint8_t *__restrict__ flags,
                                                                   const float4 *__restrict__ coef,
                                                                   const int64_t *__restrict__ blk_ofs) {
    constexpr int K = 2, SUBS = NT / 16, RB = 8;
    __shared__ SpinCoefA cf[SB];
    __shared__ float4 out[SB];  // (E, B) of the block's rows
    extern __shared__ __align__(16) unsigned char spin_smem[];
    float4 *red = reinterpret_cast<float4 *>(spin_smem);                     // [2][RB][NT]
    float4 *fw = red + 2 * RB * NT + threadIdx.x;                            // (Q, U) x (north, south): [K][2][NT]
    const int j = blockIdx.x, m = blockIdx.y, b = blockIdx.z, tid = threadIdx.x;
    const int ls = m > 2 ? m : 2, l0 = ls + SB * j, par0 = (ls - m) & 1;
    float2 *E = Eo + b * alm_stride, *B = Bo + b * alm_stride;
    if (j == 0 && m + tid < ls && m + tid <= lmax && tid < 2)  // E, B are zero for l < 2
        E[alm_idx(lmax, m + tid, m)] = B[alm_idx(lmax, m + tid, m)] = make_float2(0.f, 0.f);
    if (l0 > lmax) return;
    const int64_t np = g.npairs, blk = blk_ofs[m] + j;
    const int n = min(SB, lmax - l0 + 1);
    const uint8_t *fl = flags + blk * flag_stride(np);
    const float2 *Qf = QF + b * fm_stride + (int64_t)m * np * 2, *Uf = UF + b * fm_stride + (int64_t)m * np * 2;
#pragma unroll
    for (int i = tid; i < SB; i += NT) {
        const float4 c = i < n ? coef[blk * SB + i] : make_float4(0.f, 0.f, 0.f, 0.f);
        cf[i] = {dup2(c.x), dup2(c.y), dup2(-c.y), dup2(-c.z)};
        out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    int buf = 0;
    for (int64_t p0 = 0; p0 < np; p0 += KS * NT) {
        bool dead = true;
#pragma unroll
        for (int i = 0; i < KS * NT / 64; ++i)
            if (p0 + 64 * i < np) dead &= fl[p0 / 64 + i] == FL_DEAD;
        if (dead) continue;
        f32x2 P1, P2, M1, M2, xh, xl;
        int ep[K], em[K];
        SpinW<K> W;
        bool neg = false;
        {
            float a[6][2];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int64_t p = k < KS ? p0 + k * NT + tid : np;
                const SpinPair s = spin_state(g, m, j, p, ckP + blk * np, ckM + blk * np);
                a[0][k] = s.p1;
                a[1][k] = s.p2;
                a[2][k] = s.m1;
                a[3][k] = s.m2;
                a[4][k] = p < np ? g.pair_xhi[p] : 0.f;
                a[5][k] = p < np ? g.pair_xlo[p] : 0.f;
                ep[k] = s.ep;
                em[k] = s.em;
                neg |= (s.ep < 0) | (s.em < 0);
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f), u = q;
                if (p < np) {
                    q = load_ns(Qf + 2 * p);
                    u = load_ns(Uf + 2 * p);
                }
                fw[(2 * k) * NT] = q;
                fw[(2 * k + 1) * NT] = u;
                spin_weights(W, k, q, u, par0, s.ep >= 0, s.em >= 0);
            }
            P1 = pk(a[0][0], a[0][1]);
            P2 = pk(a[1][0], a[1][1]);
            M1 = pk(a[2][0], a[2][1]);
            M2 = pk(a[3][0], a[3][1]);
            xh = pk(a[4][0], a[4][1]);
            xl = pk(a[5][0], a[5][1]);
        }
        bool mixed = __any_sync(0xffffffffu, neg);
#pragma unroll 1
        for (int r0 = 0; r0 < n; r0 += RB, buf ^= 1) {
            float4 *rb = red + buf * RB * NT;
#pragma unroll
            for (int s = 0; s < RB; ++s) {
                const SpinCoefA c = cf[r0 + s];
                const f32x2 vp = spin_step(c.a, c.b, c.nc, xh, xl, P1, P2), vm = spin_step(c.a, c.nb, c.nc, xh, xl, M1, M2);
                P2 = P1;
                P1 = vp;
                M2 = M1;
                M1 = vm;
                float p[2], q[2];
                unpk(vp, p[0], p[1]);
                unpk(vm, q[0], q[1]);
                f32x2 e = 0, f = 0;
#pragma unroll
                for (int k = 0; k < KS; ++k) {
                    const f32x2 pd = dup2(p[k]), md = dup2(q[k]);
                    e = fma2(pd, W.pe[s & 1][k], k ? fma2(md, W.me[s & 1][k], e) : mul2(md, W.me[s & 1][k]));
                    f = fma2(pd, W.pb[s & 1][k], k ? fma2(md, W.mb[s & 1][k], f) : mul2(md, W.mb[s & 1][k]));
                }
                float4 o;
                unpk(e, o.x, o.y);
                unpk(f, o.z, o.w);
                rb[s * NT + tid] = o;
                // after every fourth row, states past 2^32 move to the next exponent (live values stay far below)
                if ((s & 3) == 3 && mixed && __any_sync(0xffffffffu, maybe_big(bits_or(bits_or(0, P1), M1)))) {
                    float a[2], d[2], fp[2], fm[2];
                    unpk(P1, a[0], a[1]);
                    unpk(M1, d[0], d[1]);
                    neg = false;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const bool up = ep[k] < 0 && fabsf(a[k]) > F32_UP, um = em[k] < 0 && fabsf(d[k]) > F32_UP;
                        fp[k] = up ? F32_DOWN : 1.f;
                        fm[k] = um ? F32_DOWN : 1.f;
                        ep[k] += up;
                        em[k] += um;
                        if ((up && ep[k] == 0) || (um && em[k] == 0))
                            spin_weights(W, k, fw[(2 * k) * NT], fw[(2 * k + 1) * NT], par0, ep[k] >= 0, em[k] >= 0);
                        neg |= (ep[k] < 0) | (em[k] < 0);
                    }
                    const f32x2 sp = pk(fp[0], fp[1]), sm = pk(fm[0], fm[1]);
                    P1 = mul2(P1, sp);
                    P2 = mul2(P2, sp);
                    M1 = mul2(M1, sm);
                    M2 = mul2(M2, sm);
                    mixed = __any_sync(0xffffffffu, neg);
                }
            }
            __syncthreads();
            // RB SUBS threads sum the buffer: the CTA's halves in turn (one of two warps at SUBS = 4)
            const int t = (tid - (buf ? RB * SUBS : 0)) & (NT - 1);
            if (t < RB * SUBS) {
                const int row = t / SUBS, sub = t % SUBS;
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float4 v = rb[row * NT + sub + i * SUBS];
                    a.x += v.x;
                    a.y += v.y;
                    a.z += v.z;
                    a.w += v.w;
                }
#pragma unroll
                for (int o = SUBS / 2; o >= 1; o >>= 1) {
                    a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
                    a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
                    a.z += __shfl_xor_sync(0xffffffffu, a.z, o);
                    a.w += __shfl_xor_sync(0xffffffffu, a.w, o);
                }
                if (sub == 0) {
                    const float4 v = out[r0 + row];
                    out[r0 + row] = make_float4(v.x + a.x, v.y + a.y, v.z + a.z, v.w + a.w);
                }
            }
        }
        __syncthreads();
    }
    __syncthreads();
#pragma unroll
    for (int i = tid; i < SB; i += NT)
        if (i < n) {
            E[alm_idx(lmax, l0 + i, m)] = make_float2(out[i].x, out[i].y);
            B[alm_idx(lmax, l0 + i, m)] = make_float2(out[i].z, out[i].w);
        }
}

// ------------------------------------------------------------------ synthesis
// With A+ = E + iB, A- = E - iB and eps = (-1)^(l-m):
//   north: Q = -1/2 sum (P A+ + M A-),      U = -i/2 sum (M A- - P A+),
//   south: Q = -1/2 sum eps (P A- + M A+),  U = -i/2 sum eps (P A- - M A+).
// P and M of one ring pair share packed instructions: the same recursion with coefficients (b, -b), and
// sums N += (P, M) (A+, A-), S += (P, M) (A-, A+), for even and odd slots apart, whose halves carry the
// separate exponents of P and M.  One warp per (group of 32 U ring pairs, order, map), as in the scalar synthesis.
struct alignas(16) SpinCoefS {  // (a, a), (b, -b), (-c, -c)
    f32x2 a, b, nc, pad;
};
struct alignas(16) SpinAlm {  // re and im of (A+, A-)
    f32x2 r, i;
};
__device__ __forceinline__ f32x2 swap2(f32x2 v) {
    float a, b;
    unpk(v, a, b);
    return pk(b, a);
}

template <int U> struct SpinS {
    f32x2 v1[U], v2[U], xh[U], xl[U];  // (P, M)
    f32x2 nr[2][U], ni[2][U], sr[2][U], si[2][U];  // [slot parity]
    int ep[U], em[U];
};

template <int U> __device__ __forceinline__ void spin_synth4(SpinS<U> &S, const SpinCoefS *cf, const SpinAlm *ac) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const SpinCoefS c = cf[s];
        const SpinAlm a = ac[s];
        const f32x2 wr = swap2(a.r), wi = swap2(a.i);
        const int q = s & 1;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const f32x2 v = spin_step(c.a, c.b, c.nc, S.xh[u], S.xl[u], S.v1[u], S.v2[u]);
            S.v2[u] = S.v1[u];
            S.v1[u] = v;
            S.nr[q][u] = fma2(v, a.r, S.nr[q][u]);
            S.ni[q][u] = fma2(v, a.i, S.ni[q][u]);
            S.sr[q][u] = fma2(v, wr, S.sr[q][u]);
            S.si[q][u] = fma2(v, wi, S.si[q][u]);
        }
    }
}

template <int U> __device__ __forceinline__ void spin_scale(SpinS<U> &S, int u, f32x2 f) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        S.nr[q][u] = mul2(S.nr[q][u], f);
        S.ni[q][u] = mul2(S.ni[q][u], f);
        S.sr[q][u] = mul2(S.sr[q][u], f);
        S.si[q][u] = mul2(S.si[q][u], f);
    }
}

template <int U, int MINB>
__global__ void __launch_bounds__(32, MINB) spin_synthesis32_kernel(GeomDev g, int lmax, int mmax, const float2 *__restrict__ E,
                                                                   const float2 *__restrict__ B, int64_t alm_stride,
                                                                   float2 *__restrict__ QG, float2 *__restrict__ UG,
                                                                   int64_t gm_stride, const float4 *__restrict__ ckP,
                                                                   const float4 *__restrict__ ckM,
                                                                   const uint8_t *__restrict__ flags,
                                                                   const float4 *__restrict__ coef,
                                                                   const int64_t *__restrict__ blk_ofs) {
    constexpr int HB = SB / 2;  // rows staged at a time: 8 KB instead of 16 per warp
    __shared__ SpinCoefS cf[HB];
    __shared__ SpinAlm ac[HB];
    const int lane = threadIdx.x, grp = blockIdx.x, m = blockIdx.y, b = blockIdx.z;
    const int ls = m > 2 ? m : 2, par0 = (ls - m) & 1;
    const int64_t np = g.npairs, fs = flag_stride(np);
    const float2 *Eb = E + b * alm_stride, *Bb = B + b * alm_stride;
    SpinS<U> S;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t p = (int64_t)(grp * U + u) * 32 + lane;
        S.xh[u] = dup2(p < np ? g.pair_xhi[p] : 0.f);
        S.xl[u] = dup2(p < np ? g.pair_xlo[p] : 0.f);
#pragma unroll
        for (int q = 0; q < 2; ++q) S.nr[q][u] = S.ni[q][u] = S.sr[q][u] = S.si[q][u] = 0;
        S.ep[u] = S.em[u] = 0;
    }
    int64_t blk = blk_ofs[m];
    for (int l0 = ls, j = 0; l0 <= lmax; l0 += SB, ++j, ++blk) {
        bool dead = true;
#pragma unroll
        for (int u = 0; u < U; u += 2) dead &= flags[blk * fs + (grp * U + u) / 2] == FL_DEAD;  // rows are padded with FL_DEAD
        if (dead) continue;
        const int n = min(SB, lmax - l0 + 1);
        bool neg = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const SpinPair s = spin_state(g, m, j, (int64_t)(grp * U + u) * 32 + lane, ckP + blk * np, ckM + blk * np);
            // the sums are in units of 2^(64 e)
            spin_scale(S, u, pk(sums_to_unit(S.ep[u], s.ep), sums_to_unit(S.em[u], s.em)));
            S.ep[u] = s.ep;
            S.em[u] = s.em;
            S.v1[u] = pk(s.p1, s.m1);
            S.v2[u] = pk(s.p2, s.m2);
            neg |= (s.ep < 0) | (s.em < 0);
        }
        bool mixed = __any_sync(0xffffffffu, neg);
        for (int h0 = 0; h0 < n; h0 += HB) {
            const int nh = min(HB, n - h0);
            __syncwarp();
#pragma unroll
            for (int k = lane; k < HB; k += 32) {
                float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
                float2 e = make_float2(0.f, 0.f), v = e;
                const int l = l0 + h0 + k;
                if (k < nh) {
                    c = coef[blk * SB + h0 + k];
                    e = Eb[alm_idx(lmax, l, m)];
                    v = Bb[alm_idx(lmax, l, m)];
                }
                cf[k] = {dup2(c.x), pk(c.y, -c.y), dup2(-c.z), 0};
                const float2 ap = make_float2(e.x - v.y, e.y + v.x), am = make_float2(e.x + v.y, e.y - v.x);
                ac[k] = {pk(ap.x, am.x), pk(ap.y, am.y)};
            }
            __syncwarp();
            int k = 0;
#pragma unroll 1
            for (; mixed && k < nh; k += 4) {
                spin_synth4(S, cf + k, ac + k);
                unsigned bits = 0;
#pragma unroll
                for (int u = 0; u < U; ++u) bits = bits_or(bits, S.v1[u]);
                if (__any_sync(0xffffffffu, maybe_big(bits))) {
                    neg = false;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        float p, q;
                        unpk(S.v1[u], p, q);
                        const bool up = S.ep[u] < 0 && fabsf(p) > F32_UP, um = S.em[u] < 0 && fabsf(q) > F32_UP;
                        const f32x2 f = pk(up ? F32_DOWN : 1.f, um ? F32_DOWN : 1.f);
                        S.v1[u] = mul2(S.v1[u], f);
                        S.v2[u] = mul2(S.v2[u], f);
                        spin_scale(S, u, f);
                        S.ep[u] += up;
                        S.em[u] += um;
                        neg |= (S.ep[u] < 0) | (S.em[u] < 0);
                    }
                    mixed = __any_sync(0xffffffffu, neg);
                }
            }
#pragma unroll 1
            for (; k < nh; k += 4) spin_synth4(S, cf + k, ac + k);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t p = (int64_t)(grp * U + u) * 32 + lane;
        if (p >= np) continue;
        spin_scale(S, u, pk(S.ep[u] == 0 ? 1.f : ldexpf(1.f, 64 * S.ep[u]), S.em[u] == 0 ? 1.f : ldexpf(1.f, 64 * S.em[u])));
        // slot parity q has l - m parity q ^ par0; (P part, M part) of north sums, and of south sums with eps
        float2 nr, ni, sr, si;
        const auto parts = [&](const f32x2 (&v)[2][U], bool south, float2 &o) {
            float2 e, d;
            unpk(par0 ? v[1][u] : v[0][u], e.x, e.y);
            unpk(par0 ? v[0][u] : v[1][u], d.x, d.y);
            if (!south) {  // (X1 + X2 of the even l - m) + (of the odd), and their difference M - P
                o = make_float2((e.x + e.y) + (d.x + d.y), (e.y - e.x) + (d.y - d.x));
            } else {
                o = make_float2((e.x + e.y) - (d.x + d.y), (e.x - e.y) - (d.x - d.y));
            }
        };
        parts(S.nr, false, nr);
        parts(S.ni, false, ni);
        parts(S.sr, true, sr);
        parts(S.si, true, si);
        const int64_t o = b * gm_stride + ((int64_t)m * np + p) * 2;
        const float h = -0.5f;
        put_ns(QG + o, h * nr.x, h * ni.x, h * sr.x, h * si.x);
        // -i/2 z = (z.im, -z.re) / 2
        put_ns(UG + o, -h * ni.y, h * nr.y, -h * si.y, h * sr.y);
    }
}

// ------------------------------------------------------------------ launches
template <int KS, int NT, int MINB>
static int run_analysis(const hb_plan *p, int nmaps, const float2 *QF, const float2 *UF, float2 *E, float2 *B, cudaStream_t st) {
    const int smem = (2 * 8 * NT + 2 * 2 * NT) * (int)sizeof(float4);
    HB_CUDA_TRY(cudaFuncSetAttribute(spin_analysis32_kernel<KS, NT, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    dim3 grid((unsigned)(p->lmax / SB + 1), (unsigned)(p->mmax + 1), (unsigned)nmaps);
    spin_analysis32_kernel<KS, NT, MINB><<<grid, NT, smem, st>>>(p->g->d, p->lmax, p->mmax, QF, UF,
                                                                 (int64_t)(p->mmax + 1) * p->g->d.npairs * 2, E, B,
                                                                 alm_size(p->lmax, p->mmax), p->ckP, p->ckM, p->ck_flags_spin,
                                                                 p->spin32, p->blk_ofs_spin);
    HB_CHECK_LAUNCH();
    return HB_OK;
}

// chunk of the sum's order: 256 pairs from 256 pairs on, 128 from 128 on, else 64
int launch_spin_analysis32(const hb_plan *p, int nmaps, const float2 *QF, const float2 *UF, float2 *E, float2 *B, cudaStream_t st) {
    const int64_t np = p->g->d.npairs;
    if (np >= 256) return run_analysis<2, 128, 5>(p, nmaps, QF, UF, E, B, st);
    if (np >= 128) return run_analysis<2, 64, 10>(p, nmaps, QF, UF, E, B, st);
    return run_analysis<1, 64, 10>(p, nmaps, QF, UF, E, B, st);
}

// Two ring pairs per lane: 2.36 ms at nside 1024; three 2.39, four 2.37 (at 12 warps per SM) to 2.55
int launch_spin_synthesis32(const hb_plan *p, int nmaps, const float2 *E, const float2 *B, float2 *QG, float2 *UG, cudaStream_t st) {
    constexpr int U = 2, MINB = 20;
    const int64_t np = p->g->d.npairs;
    dim3 grid((unsigned)((np + 32 * U - 1) / (32 * U)), (unsigned)(p->mmax + 1), (unsigned)nmaps);
    spin_synthesis32_kernel<U, MINB><<<grid, 32, 0, st>>>(p->g->d, p->lmax, p->mmax, E, B, alm_size(p->lmax, p->mmax), QG, UG,
                                                          (int64_t)(p->mmax + 1) * np * 2, p->ckP, p->ckM, p->ck_flags_spin,
                                                          p->spin32, p->blk_ofs_spin);
    HB_CHECK_LAUNCH();
    return HB_OK;
}

}  // namespace hb
