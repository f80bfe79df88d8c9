// Wigner-d matrices and the rotation of alm by Euler angles (ZYZ), FP64.
//
// Replaces the reference's rotation path (rotate_alm_euler.py:5-14 with wigner_router.py,
// wigner_fast.py and wigner_d_fast.cu:8-52; wigner_full.py:12-96; wigner_delta.py:19-56), which
// builds each d^l_{mm'}(beta) from the closed-form alternating sum.  That sum is numerically
// unusable at large l (cancellation, exp overflow), and the reference's version of it raises
// cos(beta/2) and sin(beta/2) to powers other than the textbook ones (wigner_full.py:28-37), so
// its d^l is not a rotation matrix.  Here d^l_{mm'}(beta) (d^j_{m'm} of the usual convention
// with first index m) comes from the three-term recursion in l at fixed (m, m'),
//   l R_{l+1} d_{l+1} = (2l+1) (l(l+1) cos beta - m m') d_l - (l+1) R_l d_{l-1},
//   R_l = sqrt((l^2 - m^2)(l^2 - m'^2)),
// started at l0 = max(|m|, |m'|) from the closed form of the edge element, kept as a mantissa
// and a power-of-two exponent (steps of 2^256) while it is below FP64 range.
//
// Rotation (the reference's convention, rotate_alm_euler.py / wigner_full.py:79-96):
//   a'_{lm} = sum_{m'=-l..l} exp(-i m alpha) d^l_{mm'}(beta) exp(-i m' gamma) a_{lm'},
// a_{l,-m'} = (-1)^{m'} conj(a_{lm'}) for the real field; healpy m-major layout, m >= 0 stored.
//
// Rotation kernel: R_l = s_l(m) s_l(m') with s_l(k) = sqrt(l^2 - k^2), so a step needs no root or
// division per (l, m, m').  A thread takes one m' >= 0 with both signs and MM output orders m, which
// share 1/s_l(m') and the phase-rotated input z = exp(-i m' gamma) a_{lm'}: with p = d_{m,m'}, q = (-1)^m'
// d_{m,-m'} the two signs add (p + q) Re z + i (p - q) Im z.  The factors of m are a table in shared
// memory.  Bound by issue: per l about 32 operations shared by the MM orders and 14 per order
// (a step with two roots and a division took over 100 per (l, m, m')), then the sum
// over m': TL l at a time by a transposing warp reduction (16 values per lane), one shared atomic each.
// CTAs hold chunks of 256 orders m' and add to the output with global atomics when there are
// several.  One set of alm at lmax 767: 2880 -> 609 us.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "hb_internal.cuh"
#include "hb_warp.cuh"

namespace hb {
namespace {

constexpr int ROT_NT = 256;
constexpr double TWO256 = 1.157920892373161954235709850086879078532699846656405640394575840079131296e77;  // 2^256

// d^{l0}_{m,m'}(beta), l0 = max(|m|, |m'|), for beta in [0, pi], as mantissa * 2^(256 e), from
//   d^j_{j,k} = sqrt((2j)! / ((j+k)! (j-k)!)) cos(b/2)^{j+k} (-sin(b/2))^{j-k}
// and d_{a,b} = (-1)^{a-b} d_{b,a} = d_{-b,-a}.  lc, ls: log2 cos(b/2), log2 sin(b/2) (-inf at the
// ends of the range, where the edge element is 0 or a power of 0).
__device__ __forceinline__ void d_edge(int m, int mp, double lc, double ls, double &mant, int &e) {
    int j, k, sh;
    if (abs(m) >= abs(mp)) {
        if (m >= 0) { j = m; k = mp; sh = 0; }                 // d_{l0,k}
        else { j = -m; k = -mp; sh = (mp + j) & 1; }           // d_{m,m'} = d_{-m',l0} = (-1)^{..} d_{l0,-m'}
    } else {
        if (mp > 0) { j = mp; k = m; sh = (m - j) & 1; }       // d_{m,l0} = (-1)^{m-l0} d_{l0,m}
        else { j = -mp; k = -m; sh = 0; }                      // d_{m,-l0} = d_{l0,-m}
    }
    const double l2e = 1.4426950408889634073599246810018921;  // log2 e
    double L2 = 0.5 * (lgamma(2.0 * j + 1.0) - lgamma((double)(j + k) + 1.0) - lgamma((double)(j - k) + 1.0)) * l2e;
    if (j + k > 0) L2 += (double)(j + k) * lc;
    if (j - k > 0) L2 += (double)(j - k) * ls;
    const int sign = (((j - k) & 1) ^ sh) ? -1 : 1;
    if (!(L2 > -1.0e300)) {  // -inf: an exact zero that the recursion keeps
        mant = 0.0;
        e = 0;
        return;
    }
    e = (int)floor((L2 + 128.0) / 256.0);
    mant = exp2(L2 - 256.0 * (double)e) * (double)sign;
}

// one step of the l-recursion at fixed (m, m'): (d0, d1) = (d_{l-1}, d_l) -> (d_l, d_{l+1}),
// keeping the scale exponent e (values with e < 0 are below 2^-128 of the FP64 range's middle)
__device__ __forceinline__ void d_step(int l, int m, int mp, double x, double &d0, double &d1, int &e) {
    double v;
    if (l == 0) {  // m = m' = 0: P_1 = x P_0
        v = x * d1;
    } else {
        const double dl = (double)l, m2 = (double)m * m, p2 = (double)mp * mp;
        const double R1 = sqrt(((dl + 1.0) * (dl + 1.0) - m2) * ((dl + 1.0) * (dl + 1.0) - p2));
        const double R0 = sqrt((dl * dl - m2) * (dl * dl - p2));
        v = ((2.0 * dl + 1.0) * (dl * (dl + 1.0) * x - (double)m * mp) * d1 - (dl + 1.0) * R0 * d0) / (dl * R1);
    }
    d0 = d1;
    d1 = v;
    if (e < 0 && fabs(d1) > 3.402823669209385e38) {  // 2^128: bring the scale up by 2^256
        d1 /= TWO256;
        d0 /= TWO256;
        ++e;
    }
}

// beta reduced to [0, pi]: d(beta) = d(-beta') (-1)^{m-m'} for beta = 2 pi - beta'
struct BetaRed {
    double x, lc, ls;
    bool flip;
};
__host__ __device__ __forceinline__ BetaRed beta_reduce(double beta) {
    const double twopi = 6.283185307179586476925286766559, pi = 3.141592653589793238462643383279502884;
    double b = fmod(beta, twopi);
    if (b < 0.0) b += twopi;
    BetaRed r;
    r.flip = b > pi;
    if (r.flip) b = twopi - b;
    r.x = cos(b);
    r.lc = log2(cos(0.5 * b));
    r.ls = log2(sin(0.5 * b));
    return r;
}

__global__ void __launch_bounds__(ROT_NT) wigner_d_kernel(int l, int nbeta, const double *__restrict__ beta,
                                                         double *__restrict__ out) {
    const int dim = 2 * l + 1;
    const int64_t total = (int64_t)nbeta * dim * dim;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(i / ((int64_t)dim * dim));
        const int r = (int)(i - (int64_t)b * dim * dim);
        const int m = r / dim - l, mp = r % dim - l;
        const BetaRed br = beta_reduce(beta[b]);
        double d0 = 0.0, d1;
        int e;
        d_edge(m, mp, br.lc, br.ls, d1, e);
        for (int ll = max(abs(m), abs(mp)); ll < l; ++ll) d_step(ll, m, mp, br.x, d0, d1, e);
        double v = e == 0 ? d1 : 0.0;
        if (br.flip && ((m - mp) & 1)) v = -v;
        out[i] = v;
    }
}

constexpr int ROT_V = 16;  // values per lane of the warp reduction: TL * MM * 2

// d^{l0}_{m,m'} as in d_edge, log factorials from a table
__device__ __forceinline__ void d_edge_tab(const double *lf, int m, int mp, double lc, double ls, double &mant, int &e) {
    if (!lf) return d_edge(m, mp, lc, ls, mant, e);
    int j, k, sh;
    if (m >= abs(mp)) {  // m >= 0 here
        j = m; k = mp; sh = 0;
    } else if (mp > 0) {
        j = mp; k = m; sh = (m - j) & 1;
    } else {
        j = -mp; k = -m; sh = 0;
    }
    const double l2e = 1.4426950408889634073599246810018921;  // log2 e
    double L2 = 0.5 * (lf[2 * j] - lf[j + k] - lf[j - k]) * l2e;
    if (j + k > 0) L2 += (double)(j + k) * lc;
    if (j - k > 0) L2 += (double)(j - k) * ls;
    if (!(L2 > -1.0e300)) {  // -inf: an exact zero that the recursion keeps
        mant = 0.0;
        e = 0;
        return;
    }
    e = (int)floor((L2 + 128.0) / 256.0);
    mant = exp2(L2 - 256.0 * (double)e) * ((((j - k) & 1) ^ sh) ? -1.0 : 1.0);
}

struct RotElem {  // d_{l-1}, d_l of one (m, m') and their scale exponent
    double d0, d1;
    int e;
    template <bool CLEAN> __device__ __forceinline__ void step(double t, double c) {
        const double v = fma(t, d1, -(c * d0));
        d0 = d1;
        d1 = v;
        if (CLEAN) return;
        // past 2^128 (by the high word, off the FP64 pipe): bring the scale up by 2^256
        if (e < 0 && (__double2hiint(v) & 0x7fffffff) > 0x47f00000) {
            d0 *= 0x1p-256;
            d1 *= 0x1p-256;
            ++e;
        }
    }
    __device__ __forceinline__ double value() const { return e == 0 ? d1 : 0.0; }
};

// factors of d_l = ((L(L+1) x - m m') F / s_l(m')) d_{l-1} - (C s_L(m') / s_l(m')) d_{l-2}, L = l - 1:
// F = (2L+1) / (L s_l(m)), C = (l/L) s_L(m) / s_l(m); zero for l <= m and l = 1
__device__ __forceinline__ double2 rot_factors(int l, int m) {
    const int L = l - 1;
    if (l <= m || L <= 0) return make_double2(0.0, 0.0);
    const double s2 = (double)(l - m) * (double)(l + m);
    return make_double2((2.0 * L + 1.0) / (L * sqrt(s2)), (double)l / L * sqrt((double)max(L - m, 0) * (double)(L + m) / s2));
}

// acc [lmax + 1 - mb][MM] and, with TAB, the factors of (l, m) alike and the log factorials
template <int MM, bool TAB> size_t rot_smem(int lmax) {
    return (TAB ? 32 : 16) * (size_t)MM * (size_t)(lmax + 1) + (TAB ? 8 * (size_t)(2 * lmax + 1) : 0);
}

template <int MM, bool TAB>
__global__ void __launch_bounds__(ROT_NT, 2) rotate_alm_kernel(int lmax, const double2 *__restrict__ ain,
                                                           double2 *__restrict__ aout, double alpha, double x, double lc,
                                                           double ls, int flip, double gamma, int atomic) {
    constexpr int TL = ROT_V / (2 * MM);
    extern __shared__ double2 rot_smem_buf[];
    const int mb = blockIdx.x * MM, tid = threadIdx.x, lane = tid & 31;
    const int64_t nalm = alm_idx(lmax, lmax, lmax) + 1;
    const double2 *a = ain + blockIdx.z * nalm;
    const int rows = lmax + 1 - mb;
    double2 *acc = rot_smem_buf, *fc = acc + rows * MM;
    double *lf = TAB ? reinterpret_cast<double *>(fc + rows * MM) : nullptr;
    const int mp0 = blockIdx.y * ROT_NT, lmin = max(mb, mp0);  // nothing happens below
    for (int i = tid; i < rows * MM; i += ROT_NT) {
        if (TAB) fc[i] = rot_factors(mb + i / MM, mb + i % MM);
        acc[i] = make_double2(0.0, 0.0);
    }
    if (TAB)
        for (int i = tid; i <= 2 * lmax; i += ROT_NT) lf[i] = lgamma((double)i + 1.0);
    __syncthreads();
    const int mp = mp0 + tid;
    const bool act = mp <= lmax;
    double gs, gc;
    sincos((double)mp * gamma, &gs, &gc);
    if (flip && (mp & 1)) {  // (-1)^{m-m'} of a reduced beta: the m' half of it here
        gs = -gs;
        gc = -gc;
    }
    const double qs = mp == 0 ? 0.0 : (mp & 1) ? -1.0 : 1.0;  // m' = 0 has one sign only
    RotElem P[MM], Q[MM];
#pragma unroll
    for (int i = 0; i < MM; ++i) {  // edge values, held until l passes l0 = max(m, m')
        P[i] = {0.0, 0.0, 0};
        Q[i] = {0.0, 0.0, 0};
        if (act && mb + i <= lmax) {
            d_edge_tab(lf, mb + i, mp, lc, ls, P[i].d1, P[i].e);
            d_edge_tab(lf, mb + i, -mp, lc, ls, Q[i].d1, Q[i].e);
        }
    }
    const double mp2 = (double)mp * (double)mp;
    double inv = 0.0;  // 1 / s_{l-1}(m')
    const int lw = max(lmin, __shfl_sync(0xffffffffu, mp, 0));
    const double2 *col = a + alm_idx(lmax, 0, act ? mp : 0);
    if (lw > mp) inv = rsqrt((double)(lw - 1) * (double)(lw - 1) - mp2);
    if (lw - 1 <= mp) inv = 0.0;
    // TL values of l.  CLEAN: every element of the warp is past its edge and at e = 0 (most of the range),
    // so nothing is held back, rescaled or masked.
    const auto rows_at = [&](int l0, auto clean) {
        constexpr bool CLEAN = decltype(clean)::value;
        double v[ROT_V];
#pragma unroll
        for (int s = 0; s < TL; ++s) {
            const int l = l0 + s;
            const bool on = act && (CLEAN || (l >= mp && l <= lmax));
            const double2 z0 = on ? col[l] : make_double2(0.0, 0.0);
            const double dl = (double)l, dL = dl - 1.0;
            const double i1 = CLEAN || l > mp ? rsqrt(fma(dl, dl, -mp2)) : 0.0;
            const double r = fma(dL, dL, -mp2) * inv * i1, X = dL * dl * x;  // r = s_{l-1}(m') / s_l(m')
            inv = i1;
            const double zr = fma(z0.x, gc, z0.y * gs), zi = fma(z0.y, gc, -(z0.x * gs));
#pragma unroll
            for (int i = 0; i < MM; ++i) {
                const int m = mb + i, k = (CLEAN ? l : min(l, lmax)) - mb;
                if (CLEAN || (on && l > max(m, mp))) {
                    const double2 f = TAB ? fc[k * MM + i] : rot_factors(l, m);
                    const double g = f.x * i1, c = f.y * r, mm = (double)m * (double)mp;
                    // l = 1 from l0 = 0 (m = m' = 0): P_1 = x P_0
                    P[i].template step<CLEAN>(!CLEAN && l == 1 && m == 0 && mp == 0 ? x : (X - mm) * g, c);
                    Q[i].template step<CLEAN>((X + mm) * g, c);
                }
                double *o = v + (s * MM + i) * 2;
                if (CLEAN) {
                    const double q = qs * Q[i].d1;
                    o[0] = (P[i].d1 + q) * zr;
                    o[1] = (P[i].d1 - q) * zi;
                } else {  // an input whose d is out of range does not count, infinite and NaN ones neither
                    o[0] = o[1] = 0.0;
                    if (on && l >= m && max(P[i].e, Q[i].e) == 0) {
                        const double p = P[i].value(), q = qs * Q[i].value();
                        o[0] = (p + q) * zr;
                        o[1] = (p - q) * zi;
                    }
                }
            }
        }
        const double t = warp_sums<ROT_V>(v, lane);
        const int i = lane >> 1, l = l0 + i / (2 * MM), k = (l - mb) * MM + (i / 2) % MM;
        if (!(lane & 1) && l <= lmax) atomicAdd((i & 1) ? &acc[k].y : &acc[k].x, t);
    };
    int l0 = lw;
    for (; l0 <= lmax; l0 += TL) {
        bool neg = l0 <= max(mb + MM - 1, act ? mp : 0) || l0 + TL - 1 > lmax || l0 < 2;
#pragma unroll
        for (int i = 0; i < MM; ++i) neg |= (P[i].e | Q[i].e) < 0;
        if (!__any_sync(0xffffffffu, neg)) break;
        rows_at(l0, std::false_type());
    }
    for (; l0 + TL - 1 <= lmax; l0 += TL) rows_at(l0, std::true_type());
    if (l0 <= lmax) rows_at(l0, std::false_type());
    __syncthreads();
    for (int i = tid; i < rows * MM; i += ROT_NT) {
        const int l = mb + i / MM, m = mb + i % MM;
        if (m > l || l < lmin) continue;
        double as, ac;
        sincos((double)m * alpha, &as, &ac);
        if (flip && (m & 1)) {
            as = -as;
            ac = -ac;
        }
        const double2 t = acc[i];
        double2 *o = aout + blockIdx.z * nalm + alm_idx(lmax, l, m);
        const double2 w = make_double2(t.x * ac + t.y * as, t.y * ac - t.x * as);  // times exp(-i m alpha)
        if (atomic) {
            atomicAdd(&o->x, w.x);
            atomicAdd(&o->y, w.y);
        } else {
            *o = w;
        }
    }
}

template <int MM, bool TAB>
int run_rotate(int lmax, int nmaps, const double2 *in, double2 *out, double alpha, const BetaRed &br, double gamma, cudaStream_t st) {
    const size_t smem = rot_smem<MM, TAB>(lmax);
    const int chunks = lmax / ROT_NT + 1;
    HB_CUDA_TRY(cudaFuncSetAttribute(rotate_alm_kernel<MM, TAB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     std::max((int)smem, max_smem_optin())));
    if (chunks > 1) HB_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double2) * (size_t)alm_size(lmax, lmax) * nmaps, st));
    rotate_alm_kernel<MM, TAB><<<dim3((unsigned)(lmax / MM + 1), (unsigned)chunks, (unsigned)nmaps), ROT_NT, smem, st>>>(
        lmax, in, out, alpha, br.x, br.lc, br.ls, br.flip ? 1 : 0, gamma, chunks > 1 ? 1 : 0);
    HB_CHECK_LAUNCH();
    return HB_OK;
}

}  // namespace
}  // namespace hb

using namespace hb;

extern "C" {

int hb_wigner_d(int l, int nbeta, const double *beta, double *out, hb_stream_t s) {
    if (l < 0 || l > HB_MAX_L || nbeta < 0 || (nbeta > 0 && (!beta || !out)))
        return fail(HB_ERR_INVALID, "hb_wigner_d: bad arguments");
    if (nbeta == 0) return HB_OK;
    const int64_t total = (int64_t)nbeta * (2 * l + 1) * (2 * l + 1);
    const int blocks = (int)std::min<int64_t>((total + ROT_NT - 1) / ROT_NT, 148 * 16);
    wigner_d_kernel<<<blocks, ROT_NT, 0, (cudaStream_t)s>>>(l, nbeta, beta, out);
    HB_CHECK_LAUNCH();
    return HB_OK;
}

int hb_rotate_alm(int lmax, int nmaps, const void *alm_in, void *alm_out, double alpha, double beta, double gamma,
                  hb_stream_t s) {
    if (lmax < 0 || lmax > HB_MAX_L || nmaps < 1 || nmaps > 65535 || !alm_in || !alm_out || alm_in == alm_out)
        return fail(HB_ERR_INVALID, "hb_rotate_alm: bad arguments (lmax <= 16383, out of place)");
    const BetaRed br = beta_reduce(beta);
    const auto *in = (const double2 *)alm_in;
    auto *out = (double2 *)alm_out;
    // Two orders per CTA while the tables fit (lmax <= 2800), else one, without tables where they do not
    // fit either.  At lmax 767 two orders take 609 us; compared with four orders, 635 against 676 us (both at two
    // CTAs per SM, before the input's gate was predicated).
    const auto st = (cudaStream_t)s;
    if (rot_smem<2, true>(lmax) <= 220 * 1024) return run_rotate<2, true>(lmax, nmaps, in, out, alpha, br, gamma, st);
    if (rot_smem<1, true>(lmax) <= 220 * 1024) return run_rotate<1, true>(lmax, nmaps, in, out, alpha, br, gamma, st);
    return run_rotate<1, false>(lmax, nmaps, in, out, alpha, br, gamma, st);
}

}  // extern "C"
