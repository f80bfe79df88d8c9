// Scalar Legendre kernels in FP32 (the FP64 ones are in hb_legendre.cu), and the launchers of both.
//
// Lambda is generated in registers by the normalised recursion
//     lambda_l = A_l x lambda_{l-1} + B_l lambda_{l-2},
//     A_l = sqrt((4l^2-1)/(l^2-m^2)),  B_l = -A_l sqrt(((l-1)^2-m^2)/(4(l-1)^2-1)),
// and contracted at once, never stored; the north and south rings of a pair are folded into
// E = F_N + F_S (even l-m) and O = F_N - F_S (odd l-m).  x is carried as a float pair (hi + lo): a
// rounded cos(theta) shifts a ring by ~1e-7/sin(theta) rad, an l*dtheta phase error that reaches
// 1e-4 at l ~ 4000.  The recursion restarts every 256 l from the plan's FP64-computed checkpoints;
// its start values lambda_mm = (-1)^m sqrt((2m+1)!!/((2m)!! 4pi)) sin^m theta come from FP64 log2
// tables.  States are mantissa * 2^(64 e): while e < 0 (|lambda| < 2^-32) a value counts as zero in the
// analysis, and every 4 l a state past 2^32 moves to the next exponent.
//
// What bounds the kernels: the FMA pipe, 6 operations per (l, ring pair) for one map (4 of them the
// recursion, shared by the NB maps of a CTA).  Two ring pairs share each packed instruction, which
// leaves half the issue slots to loads and reductions; blocks of 256 l in which a set of pairs stays
// evanescent are skipped by the plan's flags (a quarter of the work at lmax = 2 nside).
// One map at nside 1024, lmax 2047: synthesis 1636 -> 813 us (73 % FMA pipe), analysis 2000 -> 1320 us
// (51 %; following the pairs that leave e < 0 within a block takes 160 us of it).  The arithmetic and the
// order of every sum of the analysis are unchanged (same bits).
#include <cmath>

#include "hb_f32x2.cuh"
#include "hb_internal.cuh"

namespace hb {

constexpr int LB = 256;  // l per block (the checkpoint spacing)

// start value lambda_mm = mant * 2^(64 e)
__device__ __forceinline__ void sectoral_start32(const GeomDev &g, int m, int64_t p, float &mant, int &e) {
    const double L = g.log2cm[m] + (double)m * g.pair_log2sin[p];
    e = (int)floor((L + 32.0) / 64.0);
    const double v = exp2(L - 64.0 * e);
    mant = (float)((m & 1) ? -v : v);
}

// one recursion step of two pairs: (l1, l2) = (lambda_{l-1}, lambda_{l-2}) -> lambda_l
__device__ __forceinline__ f32x2 lambda_step(f32x2 A, f32x2 B, f32x2 xh, f32x2 xl, f32x2 l1, f32x2 l2) {
    return fma2(B, l2, mul2(A, fma2(xh, l1, mul2(xl, l1))));
}

// state of pair p at the first l of block j (lambda_{l0-1}, lambda_{l0-2}, e); zero past the last pair
__device__ __forceinline__ void block_state(const GeomDev &g, int m, int j, int64_t p, const float4 *ckrow, float &l1, float &l2,
                                            int &e) {
    l1 = l2 = 0.f;
    e = 0;
    if (p >= g.npairs) return;
    if (j == 0) {
        sectoral_start32(g, m, p, l2, e);
    } else {
        const float4 c = ckrow[p];
        l1 = c.x;
        l2 = c.y;
        e = __float_as_int(c.z);
    }
}

// whether a pair that starts a block with e < 0 keeps e < 0 through it, by the next block's checkpoint row
__device__ __forceinline__ bool stays_dead(const float4 *next, int64_t p) { return __float_as_int(next[p].z) < 0; }

struct alignas(16) Coef2 {  // (A_l, B_l), each in both halves
    f32x2 a, b;
};

// ------------------------------------------------------------------ analysis
// a_lm = sum over pairs of lambda_l (E or O).  One CTA per (block of 256 l, order, NB maps): blocks
// are independent (each restarts from its checkpoints), x runs fastest so that the blocks of an
// order find F(m) in L2, and each CTA writes its alm alone, without atomics.
//
// The sum over a chunk of K NT pairs runs in a fixed order: thread t < NT adds its K pairs k NT + t,
// columns t = s + SUBS j add up over j = 0 .. 15 (through shared memory, RB rows at a time, double
// buffered), and the SUBS = NT / 16 results form a binary tree (shuffles).  The recursion is packed over
// the pairs k and k + 1 of a thread; their contraction is two scalar operations each, since the sum
// runs through them in turn.
template <int K, int NB> struct AState {
    f32x2 l1[K / 2], l2[K / 2], xh[K / 2], xl[K / 2];
    float er[NB][K], ei[NB][K], qr[NB][K], qi[NB][K];  // zero while e < 0
    int e[K];
};

// (E, O) of a ring pair from its (north, south) coefficients
template <int K, int NB> __device__ __forceinline__ void set_weights(AState<K, NB> &S, int u, int b, float4 f) {
    S.er[b][u] = f.x + f.z;
    S.ei[b][u] = f.y + f.w;
    S.qr[b][u] = f.x - f.z;
    S.qi[b][u] = f.y - f.w;
}

template <int U0, int K, int NB, int NT>
__device__ __forceinline__ void anal_step4(AState<K, NB> &S, const Coef2 *cf, float2 *red) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const Coef2 c = cf[s];
        float ar[NB], ai[NB];
#pragma unroll
        for (int u = U0; u < K; u += 2) {
            const f32x2 v2 = lambda_step(c.a, c.b, S.xh[u / 2], S.xl[u / 2], S.l1[u / 2], S.l2[u / 2]);
            S.l2[u / 2] = S.l1[u / 2];
            S.l1[u / 2] = v2;
            float v[2];
            unpk(v2, v[0], v[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const float wr = s & 1 ? S.qr[b][u + h] : S.er[b][u + h], wi = s & 1 ? S.qi[b][u + h] : S.ei[b][u + h];
                    ar[b] = u + h == U0 ? v[h] * wr : fmaf(v[h], wr, ar[b]);
                    ai[b] = u + h == U0 ? v[h] * wi : fmaf(v[h], wi, ai[b]);
                }
            }
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) red[(s * NB + b) * NT] = make_float2(ar[b], ai[b]);
    }
}

// Moves to the next exponent after every fourth row, in the pair sets up to um (the last one with e < 0
// in the warp).  A pair that reaches e = 0 gets its weights from the thread's column fw of the staged
// (north, south) coefficients.
template <int U0, int K, int NB, int NT> __device__ __forceinline__ void anal_rescale(AState<K, NB> &S, int um, const float4 *fw) {
#pragma unroll
    for (int u = U0; u < K; u += 2) {
        if (u > um) break;
        // live values stay far below 2^32, so a larger one has e < 0
        if (!__any_sync(0xffffffffu, maybe_big(bits_or(0, S.l1[u / 2])))) continue;
        float v[2], f[2] = {1.f, 1.f};
        unpk(S.l1[u / 2], v[0], v[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (S.e[u + h] < 0 && fabsf(v[h]) > F32_UP) {
                f[h] = F32_DOWN;
                if (++S.e[u + h] == 0) {
#pragma unroll
                    for (int b = 0; b < NB; ++b) set_weights(S, u + h, b, fw[((u + h) * NB + b) * NT]);
                }
            }
        S.l1[u / 2] = mul2(S.l1[u / 2], pk(f[0], f[1]));
        S.l2[u / 2] = mul2(S.l2[u / 2], pk(f[0], f[1]));
    }
}

// last even u whose pair sets u, u + 1 hold an e < 0 in the warp (-1: none)
template <int U0, int K, int NB> __device__ __forceinline__ int last_negative(const AState<K, NB> &S) {
    int um = -1;
#pragma unroll
    for (int u = U0; u < K; u += 2)
        if (__any_sync(0xffffffffu, (S.e[u] | S.e[u + 1]) < 0)) um = u;
    return um;
}

// Rows 0 .. n-1 of the block for the pair sets U0 .. K-1 (the sets before them are evanescent).  Item
// (row, map) of a buffer is summed by SUBS threads into out[item] (every item has one writer).
template <int U0, int K, int NB, int NT>
__device__ __forceinline__ void anal_rows(AState<K, NB> &S, const Coef2 *cf, float2 *red, const float4 *fw, float2 *out, int n) {
    constexpr int SUBS = NT / 16, RB = 16 / NB;
    const int tid = threadIdx.x, item = tid / SUBS, sub = tid % SUBS;
    int um = last_negative<U0>(S);
    for (int r0 = 0; r0 < n; r0 += RB, cf += RB) {
        float2 *buf = red + ((r0 / RB) & 1) * RB * NB * NT;
#pragma unroll
        for (int s = 0; s < RB; s += 4) {
            anal_step4<U0, K, NB, NT>(S, cf + s, buf + s * NB * NT + tid);
            if (um >= 0) anal_rescale<U0, K, NB, NT>(S, um, fw);
        }
        if (um >= 0) um = last_negative<U0>(S);
        __syncthreads();
        float rr = 0.f, ri = 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float2 v = buf[item * NT + sub + j * SUBS];
            rr += v.x;
            ri += v.y;
        }
#pragma unroll
        for (int o = SUBS / 2; o >= 1; o >>= 1) {
            rr += __shfl_xor_sync(0xffffffffu, rr, o);
            ri += __shfl_xor_sync(0xffffffffu, ri, o);
        }
        if (sub == 0) out[r0 * NB + item] = cadd(out[r0 * NB + item], make_float2(rr, ri));
    }
}

template <int U0, int K, int NB, int NT>
__device__ __forceinline__ void anal_from(int u0, AState<K, NB> &S, const Coef2 *cf, float2 *red, const float4 *fw,
                                          float2 *out, int n) {
    if (u0 < U0 + 2)
        anal_rows<U0, K, NB, NT>(S, cf, red, fw, out, n);
    else if constexpr (U0 + 2 < K)
        anal_from<U0 + 2, K, NB, NT>(u0, S, cf, red, fw, out, n);
}

// KS: pairs per thread of the sum's order (K, or 1 when K = 2 stands for it)
template <int K, int KS, int NT, int NB, int MINB>
__global__ void __launch_bounds__(NT, MINB) leg_analysis32_kernel(GeomDev g, int lmax, int mmax, const float2 *__restrict__ Fm,
                                                                  int64_t fm_stride, float2 *__restrict__ alm,
                                                                  int64_t alm_stride, const float4 *__restrict__ ck,
                                                                  const uint8_t *__restrict__ flags,
                                                                  const float2 *__restrict__ coef,
                                                                  const int64_t *__restrict__ blk_ofs,
                                                                  const int32_t *__restrict__ mlist) {
    __shared__ Coef2 cf[LB];
    __shared__ float2 out[LB * NB];
    extern __shared__ __align__(16) unsigned char leg_smem[];
    float2 *red = reinterpret_cast<float2 *>(leg_smem);  // [2][16 / NB rows][NB][NT], then F: [K][NB][NT]
    float4 *fw = reinterpret_cast<float4 *>(red + 2 * 16 * NT) + threadIdx.x;
    const int j = blockIdx.x, tid = threadIdx.x;
    // F row blockIdx.y holds order m (all orders, or the orders of mlist in list order)
    const int m = mlist ? mlist[blockIdx.y] : blockIdx.y, l0 = m + LB * j;
    if (m < 0 || m > mmax || l0 > lmax) return;  // a listed order outside the plan: nothing read or written
    const int64_t np = g.npairs, blk = blk_ofs[m] + j;
    const int n = min(LB, lmax - l0 + 1);
    const float4 *ckrow = ck + blk * np, *cknext = blk + 1 < blk_ofs[m + 1] ? ckrow + np : nullptr;
    const uint8_t *fl = flags + blk * flag_stride(np);
    const float2 *F = Fm + (int64_t)blockIdx.z * NB * fm_stride + (int64_t)blockIdx.y * np * 2;
#pragma unroll
    for (int i = tid; i < LB; i += NT) {
        const float2 c = i < n ? coef[blk * LB + i] : make_float2(0.f, 0.f);
        cf[i] = {dup2(c.x), dup2(c.y)};
    }
#pragma unroll
    for (int i = tid; i < LB * NB; i += NT) out[i] = make_float2(0.f, 0.f);
    __syncthreads();
    for (int64_t p0 = 0; p0 < np; p0 += KS * NT) {
        int u0 = K;  // first set of NT pairs that does not stay evanescent
#pragma unroll
        for (int u = KS - 1; u >= 0; --u) {
            bool dead = true;
#pragma unroll
            for (int i = 0; i < NT / 64; ++i) {
                const int64_t f = (p0 + u * NT) / 64 + i;
                if (f * 64 < np) dead &= fl[f] == FL_DEAD;
            }
            if (!dead) u0 = u;
        }
        if (u0 == K) continue;
        AState<K, NB> S;
#pragma unroll
        for (int u = 0; u < K; u += 2) {
            float a1[2], a2[2], xh[2], xl[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int64_t p = u + i < KS ? p0 + (u + i) * NT + tid : np;
                block_state(g, m, j, p, ckrow, a1[i], a2[i], S.e[u + i]);
                xh[i] = p < np ? g.pair_xhi[p] : 0.f;
                xl[i] = p < np ? g.pair_xlo[p] : 0.f;
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);  // (north, south)
                    if (p < np) f = load_ns(F + b * fm_stride + 2 * p);
                    fw[((u + i) * NB + b) * NT] = f;
                    set_weights(S, u + i, b, S.e[u + i] < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : f);
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)  // evanescent over the whole block: no values, and no exponent to follow
                if (S.e[u + i] < 0 && cknext && stays_dead(cknext, p0 + (u + i) * NT + tid)) {
                    a1[i] = a2[i] = 0.f;
                    S.e[u + i] = 0;
                }
            S.l1[u / 2] = pk(a1[0], a1[1]);
            S.l2[u / 2] = pk(a2[0], a2[1]);
            S.xh[u / 2] = pk(xh[0], xh[1]);
            S.xl[u / 2] = pk(xl[0], xl[1]);
        }
        anal_from<0, K, NB, NT>(u0, S, cf, red, fw, out, n);
        __syncthreads();
    }
    __syncthreads();
#pragma unroll
    for (int i = tid; i < LB * NB; i += NT) {
        const int r = i / NB;
        if (r < n) alm[((int64_t)blockIdx.z * NB + i % NB) * alm_stride + alm_idx(lmax, l0 + r, m)] = out[i];
    }
}

// ------------------------------------------------------------------ synthesis
// G_N/S(m) = sum_l a_lm lambda_lm (+-1)^(l-m).  One warp per (group of 64 U ring pairs, order, NB maps)
// with the sums in registers; single warps, because the warps of larger CTAs would wait for each
// other at every block (those near the pole skip most of them).  The sums are kept in units of
// 2^(64 e).
template <int U, int NB> struct SState {
    f32x2 l1[U], l2[U], xh[U], xl[U];
    f32x2 ar[2][NB][U], ai[2][NB][U];  // even and odd l - m
    int e[U][2];
};

template <int U, int NB> __device__ __forceinline__ void synth4(SState<U, NB> &S, const Coef2 *cf, const float2 *ac) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const Coef2 c = cf[s];
        f32x2 a[NB], b[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const float2 v = ac[i * LB + s];
            a[i] = dup2(v.x);
            b[i] = dup2(v.y);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const f32x2 v = lambda_step(c.a, c.b, S.xh[u], S.xl[u], S.l1[u], S.l2[u]);
            S.l2[u] = S.l1[u];
            S.l1[u] = v;
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                S.ar[s & 1][i][u] = fma2(v, a[i], S.ar[s & 1][i][u]);
                S.ai[s & 1][i][u] = fma2(v, b[i], S.ai[s & 1][i][u]);
            }
        }
    }
}

template <int U, int NB> __device__ __forceinline__ void scale_sums(SState<U, NB> &S, int u, f32x2 f) {
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            S.ar[q][i][u] = mul2(S.ar[q][i][u], f);
            S.ai[q][i][u] = mul2(S.ai[q][i][u], f);
        }
}

template <int U, int NB, int MINB>
__global__ void __launch_bounds__(32, MINB) leg_synthesis32_kernel(GeomDev g, int lmax, int mmax, const float2 *__restrict__ alm,
                                                                  int64_t alm_stride, float2 *__restrict__ Gm, int64_t gm_stride,
                                                                  const float4 *__restrict__ ck, const uint8_t *__restrict__ flags,
                                                                  const float2 *__restrict__ coef,
                                                                  const int64_t *__restrict__ blk_ofs,
                                                                  const int32_t *__restrict__ mlist) {
    __shared__ Coef2 cf[LB];
    __shared__ float2 ac[NB * LB];
    const int lane = threadIdx.x, grp = blockIdx.x;
    // G row blockIdx.y holds order m (all orders, or the orders of mlist in list order)
    const int m = mlist ? mlist[blockIdx.y] : blockIdx.y;
    if (m < 0 || m > mmax) return;  // a listed order outside the plan: nothing read or written
    const int64_t np = g.npairs, fs = flag_stride(np);
    const float2 *a = alm + (int64_t)blockIdx.z * NB * alm_stride;
    SState<U, NB> S;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        float xh[2], xl[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int64_t p = (int64_t)(grp * U + u) * 64 + 2 * lane + i;
            xh[i] = p < np ? g.pair_xhi[p] : 0.f;
            xl[i] = p < np ? g.pair_xlo[p] : 0.f;
            S.e[u][i] = 0;
        }
        S.xh[u] = pk(xh[0], xh[1]);
        S.xl[u] = pk(xl[0], xl[1]);
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int i = 0; i < NB; ++i) S.ar[q][i][u] = S.ai[q][i][u] = 0;
    }
    int64_t blk = blk_ofs[m];
    for (int l0 = m, j = 0; l0 <= lmax; l0 += LB, ++j, ++blk) {
        bool dead = true;
#pragma unroll
        for (int u = 0; u < U; ++u) dead &= flags[blk * fs + grp * U + u] == FL_DEAD;  // rows are padded with FL_DEAD
        if (dead) continue;
        const int n = min(LB, lmax - l0 + 1);
        __syncwarp();
#pragma unroll
        for (int k = lane; k < LB; k += 32) {
            const float2 c = k < n ? coef[blk * LB + k] : make_float2(0.f, 0.f);
            cf[k] = {dup2(c.x), dup2(c.y)};
#pragma unroll
            for (int i = 0; i < NB; ++i)
                ac[i * LB + k] = k < n ? a[i * alm_stride + alm_idx(lmax, l0 + k, m)] : make_float2(0.f, 0.f);
        }
        bool neg = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float l1[2], l2[2], f[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                int e;
                block_state(g, m, j, (int64_t)(grp * U + u) * 64 + 2 * lane + i, ck + blk * np, l1[i], l2[i], e);
                f[i] = sums_to_unit(S.e[u][i], e);
                S.e[u][i] = e;
                neg |= e < 0;
            }
            scale_sums(S, u, pk(f[0], f[1]));
            S.l1[u] = pk(l1[0], l1[1]);
            S.l2[u] = pk(l2[0], l2[1]);
        }
        bool mixed = __any_sync(0xffffffffu, neg);
        __syncwarp();
        int k = 0;
#pragma unroll 1
        for (; mixed && k < n; k += 4) {
            synth4(S, cf + k, ac + k);
            unsigned bits = 0;
#pragma unroll
            for (int u = 0; u < U; ++u) bits = bits_or(bits, S.l1[u]);
            if (__any_sync(0xffffffffu, maybe_big(bits))) {
                neg = false;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    float x, y;
                    unpk(S.l1[u], x, y);
                    const bool ux = S.e[u][0] < 0 && fabsf(x) > F32_UP, uy = S.e[u][1] < 0 && fabsf(y) > F32_UP;
                    const f32x2 f = pk(ux ? F32_DOWN : 1.f, uy ? F32_DOWN : 1.f);
                    S.l1[u] = mul2(S.l1[u], f);
                    S.l2[u] = mul2(S.l2[u], f);
                    scale_sums(S, u, f);
                    S.e[u][0] += ux;
                    S.e[u][1] += uy;
                    neg |= (S.e[u][0] < 0) | (S.e[u][1] < 0);
                }
                mixed = __any_sync(0xffffffffu, neg);
            }
        }
#pragma unroll 1
        for (; k < n; k += 4) synth4(S, cf + k, ac + k);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            float er[2], ei[2], qr[2], qi[2];
            unpk(S.ar[0][i][u], er[0], er[1]);
            unpk(S.ai[0][i][u], ei[0], ei[1]);
            unpk(S.ar[1][i][u], qr[0], qr[1]);
            unpk(S.ai[1][i][u], qi[0], qi[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t p = (int64_t)(grp * U + u) * 64 + 2 * lane + h;
                if (p >= np) continue;
                const float f = S.e[u][h] == 0 ? 1.f : ldexpf(1.f, 64 * S.e[u][h]);
                float2 *G = Gm + ((int64_t)blockIdx.z * NB + i) * gm_stride + ((int64_t)blockIdx.y * np + p) * 2;
                put_ns(G, (er[h] + qr[h]) * f, (ei[h] + qi[h]) * f, (er[h] - qr[h]) * f, (ei[h] - qi[h]) * f);
            }
        }
}

// ------------------------------------------------------------------ launches
struct Leg32 {
    const hb_plan *p;
    int rows;
    const int32_t *mlist;
    cudaStream_t st;
    int64_t np() const { return p->g->d.npairs; }
    int64_t f_stride() const { return (int64_t)rows * np() * 2; }
    int64_t a_stride() const { return alm_size(p->lmax, p->mmax); }
};

template <int K, int KS, int NT, int NB, int MINB> static int run_analysis(const Leg32 &L, int nz, const float2 *F, float2 *alm) {
    const int smem = 2 * 16 * NT * (int)sizeof(float2) + K * NB * NT * (int)sizeof(float4);
    HB_CUDA_TRY(cudaFuncSetAttribute(leg_analysis32_kernel<K, KS, NT, NB, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    dim3 grid((unsigned)(L.p->lmax / LB + 1), (unsigned)L.rows, (unsigned)nz);
    leg_analysis32_kernel<K, KS, NT, NB, MINB><<<grid, NT, smem, L.st>>>(L.p->g->d, L.p->lmax, L.p->mmax, F, L.f_stride(), alm,
                                                                         L.a_stride(), L.p->ck, L.p->ck_flags, L.p->leg32,
                                                                         L.p->blk_ofs, L.mlist);
    HB_CHECK_LAUNCH();
    return HB_OK;
}
template <int U, int NB, int MINB> static int run_synthesis(const Leg32 &L, int nz, const float2 *alm, float2 *G) {
    dim3 grid((unsigned)((L.np() + 64 * U - 1) / (64 * U)), (unsigned)L.rows, (unsigned)nz);
    leg_synthesis32_kernel<U, NB, MINB><<<grid, 32, 0, L.st>>>(L.p->g->d, L.p->lmax, L.p->mmax, alm, L.a_stride(), G, L.f_stride(),
                                                               L.p->ck, L.p->ck_flags, L.p->leg32, L.p->blk_ofs, L.mlist);
    HB_CHECK_LAUNCH();
    return HB_OK;
}

// The number of pairs decides how the analysis orders its sum (columns of K pairs, NT columns): one chunk of 512
// up to 512 pairs and of 1024 up to 1024, chunks of 2048 above, of 128 and 64 below 256 pairs.  In us, chunks of 512 /
// 1024 / 2048, lmax equal to the pairs: 600 pairs, one map 100 / 88 / 134, two 142 / 119 / 252; 1000, 226 / 232 / 344, two
// 334 / 317 / 670; lmax 1.5 times the pairs: 600, 182 / 182 / 274; 1000, 442 / 495 / 733; 2048, 2940 / 3237 / 2794.  Chunks of
// 2048 leave no registers for a second map's weights, so their maps run singly.
template <int NB> static int analysis_nb(const Leg32 &L, int nz, const float2 *F, float2 *alm) {
    if (L.np() > 1024) return run_analysis<8, 8, 256, 1, 2>(L, nz * NB, F, alm);
    if (L.np() > 512) return run_analysis<4, 4, 256, NB, 2>(L, nz, F, alm);
    if (L.np() >= 256) return run_analysis<4, 4, 128, NB, 5>(L, nz, F, alm);
    if (L.np() >= 64) return run_analysis<2, 2, 64, NB, 10>(L, nz, F, alm);
    return run_analysis<2, 1, 64, NB, 10>(L, nz, F, alm);
}
template <int NB> static int synthesis_nb(const Leg32 &L, int nz, const float2 *alm, float2 *G) {
    if (L.np() >= 512) return run_synthesis<2, NB, NB == 1 ? 20 : 16>(L, nz, alm, G);
    return run_synthesis<1, NB, 20>(L, nz, alm, G);
}

// Maps in pairs that share one recursion; below 256 ring pairs one launch of single maps, which are
// bound by latency there.
template <typename Fn2, typename Fn1> static int by_two(int nmaps, int64_t np, Fn2 f2, Fn1 f1) {
    const int n2 = np >= 256 ? nmaps / 2 : 0;
    if (n2)
        if (int rc = f2(n2, 0)) return rc;
    return nmaps > 2 * n2 ? f1(nmaps - 2 * n2, 2 * n2) : HB_OK;
}
static int analysis32(const hb_plan *p, int nmaps, const float2 *F, float2 *alm, cudaStream_t st, int nm, const int32_t *mlist) {
    const Leg32 L{p, mlist ? nm : p->mmax + 1, mlist, st};
    const int64_t fs = L.f_stride(), as = L.a_stride();
    return by_two(nmaps, L.np(), [&](int nz, int b) { return analysis_nb<2>(L, nz, F + b * fs, alm + b * as); },
                  [&](int nz, int b) { return analysis_nb<1>(L, nz, F + b * fs, alm + b * as); });
}
static int synthesis32(const hb_plan *p, int nmaps, const float2 *alm, float2 *G, cudaStream_t st, int nm, const int32_t *mlist) {
    const Leg32 L{p, mlist ? nm : p->mmax + 1, mlist, st};
    const int64_t fs = L.f_stride(), as = L.a_stride();
    return by_two(nmaps, L.np(), [&](int nz, int b) { return synthesis_nb<2>(L, nz, alm + b * as, G + b * fs); },
                  [&](int nz, int b) { return synthesis_nb<1>(L, nz, alm + b * as, G + b * fs); });
}

int launch_leg_analysis64(const hb_plan *p, int nmaps, const double2 *F, double2 *alm, cudaStream_t st, int nm,
                          const int32_t *mlist);
int launch_leg_synthesis64(const hb_plan *p, int nmaps, const double2 *alm, double2 *G, cudaStream_t st, int nm,
                           const int32_t *mlist);

int launch_leg_analysis(const hb_plan *p, int precision, int nmaps, const void *Fm, void *alm, cudaStream_t st, int nm,
                        const int32_t *mlist) {
    HB_NVTX("legendre_analysis");
    if (precision == 32) return analysis32(p, nmaps, (const float2 *)Fm, (float2 *)alm, st, nm, mlist);
    return launch_leg_analysis64(p, nmaps, (const double2 *)Fm, (double2 *)alm, st, nm, mlist);
}

int launch_leg_synthesis(const hb_plan *p, int precision, int nmaps, const void *alm, void *Gm, cudaStream_t st, int nm,
                         const int32_t *mlist) {
    HB_NVTX("legendre_synthesis");
    if (precision == 32) return synthesis32(p, nmaps, (const float2 *)alm, (float2 *)Gm, st, nm, mlist);
    return launch_leg_synthesis64(p, nmaps, (const double2 *)alm, (double2 *)Gm, st, nm, mlist);
}

}  // namespace hb
