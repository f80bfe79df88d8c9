// Transform plans: a geometry plus (lmax, mmax) plus the FP64-computed recursion checkpoints
// that re-anchor the FP32 Legendre recursions.
//
// Why: in FP32 the three-term recursion lambda_l = A_l x lambda_{l-1} + B_l lambda_{l-2}
// accumulates rounding error linearly in l near the poles (where x -> 1 the recursion's
// characteristic roots merge), reaching ~1e-4 relative at l ~ 4000 for small m.  The plan stores,
// for every m, every block of R = 256 consecutive l and every ring pair, the recursion state
// (lambda_{l0-1}, lambda_{l0-2}) at the block start l0, computed by the same recursion in FP64
// and rounded to the FP32 kernels' scaled format (mantissa pair + power-of-2^64 exponent).  The
// FP32 kernels reload it at each block start, so FP32 error can only accumulate over R steps.
// The same table lets a kernel start the recursion at any block (used by the batched path).
//
// Layout: ck[(blk_ofs[m] + j) * npairs + p] = float4(mu1, mu2, bits(e), 0) for block j of m
// (block j starts at l = m + j*R for the scalar recursion, at l = max(m,2) + j*R for spin-2).
// Each row of the scalar table has a flag byte per 64 pairs (hb_internal.cuh) by which the FP32
// kernels skip blocks that stay evanescent.
//
// Plans for FP64 calls (all without HB_PLAN_NO_FP64) hold the FP64 coefficient tables of the scalar
// recursions (LegTab): their scale factors are products over l, which a kernel would have to rebuild per
// CTA (48 bytes per (l, m), 0.4 GB at lmax 4095).  FP32 plans hold the one-step coefficients (8 bytes per
// (l, m)).
#include <cmath>
#include <vector>

#include "hb_internal.cuh"

namespace hb {

// (A_l, B_l) of the scalar recursion in FP64 (l > m)
__device__ __forceinline__ void ck_scalar_coef(int l, int m, double &A, double &B) {
    double ll = l, mm = m;
    A = sqrt((4.0 * ll * ll - 1.0) / ((ll - mm) * (ll + mm)));
    B = (l - 1 > m) ? -A * sqrt(((ll - 1.0 - mm) * (ll - 1.0 + mm)) / (4.0 * (ll - 1.0) * (ll - 1.0) - 1.0)) : 0.0;
}

// Convert an FP64 scaled state (v1, v2) * 2^(512 e) to the FP32 format (mu1, mu2) * 2^(64 ef).  The exponent
// is that of the larger value: one alone can be near zero on an oscillating pair (every second value on a
// ring at the equator), and such a pair is live.
__device__ __forceinline__ float4 to_f32_state(double v1, double v2, int e) {
    const double ref = fmax(fabs(v1), fabs(v2));
    if (ref == 0.0) return make_float4(0.f, 0.f, __int_as_float(0), 0.f);
    int ex;
    frexp(ref, &ex);  // |ref| in [2^(ex-1), 2^ex)
    double L = (double)ex + 512.0 * (double)e;
    int ef = (int)floor((L + 32.0) / 64.0);
    if (ef > 0) ef = 0;
    long long sh = 512LL * e - 64LL * ef;
    int shi = (int)(sh < -2000 ? -2000 : (sh > 2000 ? 2000 : sh));
    return make_float4((float)ldexp(v1, shi), (float)ldexp(v2, shi), __int_as_float(ef), 0.f);
}

// eps_l = sqrt((l^2 - m^2) / (4 l^2 - 1))
__device__ __forceinline__ double leg_eps(int l, int m) {
    const double ll = l, mm = m;
    return sqrt((ll - mm) * (ll + mm) / ((2.0 * ll - 1.0) * (2.0 * ll + 1.0)));
}

// LegTab rows of one order per thread.  N_k and M_l follow from their neighbours' products
// N_k N_{k+1} eps_{l+2} eps_{l+3} = 1/4 and M_l M_{l+1} eps_{l+1} = 1/2; the free first values are
// the smooth ones, so that both stay of order one.
__global__ void leg_table_kernel(int lmax, int mmax, LegTab tb) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m > mmax) return;
    double e1 = leg_eps(m + 1, m), e2 = leg_eps(m + 2, m);
    double N = sqrt(0.25 / (e1 * e2)), M = sqrt(0.5 / e1), Mprev = 0.0;
    double *t = tb.row(m, 0);
    for (int k = 0, l = m; l <= lmax; ++k, l += 2, t += LT_N) {
        const double e3 = leg_eps(l + 3, m), a = 4.0 * N * N, M1 = 0.5 / (e1 * M), sg = (k & 1) ? -1.0 : 1.0;
        t[LT_A] = a;
        t[LT_G] = a * (1.0 - e1 * e1 - e2 * e2) - 2.0;
        t[LT_P] = N * e1;
        t[LT_Q] = l + 2 <= lmax ? N * e2 : 0.0;
        t[LT_NX] = l + 1 <= lmax ? N : 0.0;
        t[LT_B0] = -2.0 * Mprev * Mprev;
        t[LT_B1] = 2.0 * M * M;
        t[LT_M0] = sg * M;
        t[LT_M1] = sg * M1;
        for (int i = LT_NX + 1; i < LT_N; ++i) t[i] = 0.0;
        N = 0.25 / (e2 * e3 * N);
        Mprev = M1;
        M = 0.5 / (e2 * M1);
        e1 = e3;
        e2 = leg_eps(l + 4, m);
    }
}

constexpr int CKR = 256;   // checkpoint block length (== COEF_CH of the Legendre kernels)
constexpr int CK_NT = 128;

// (A_l, B_l) of the FP32 kernels, zero past lmax; l = m gives (0, 1): the first block's state is
// (0, lambda_mm)
__global__ void leg32_coef_kernel(int lmax, const int64_t *__restrict__ blk_ofs, float2 *__restrict__ tab) {
    const int m = blockIdx.x;
    float2 *t = tab + blk_ofs[m] * CKR;
    const int64_t n = (blk_ofs[m + 1] - blk_ofs[m]) * CKR;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        double A = 0.0, B = i == 0 ? 1.0 : 0.0;
        if (i > 0 && m + i <= lmax) ck_scalar_coef(m + (int)i, m, A, B);
        t[i] = make_float2((float)A, (float)B);
    }
}


// one row of the flag table: the CTA's CK_NT / 64 units, the last CTA of a row also its padding
__device__ __forceinline__ void write_flags(uint8_t *flags, int64_t row, int64_t np, const int *any_neg, const int *any_live) {
    const int64_t stride = flag_stride(np), unit = (int64_t)blockIdx.y * (CK_NT / 64) + threadIdx.x;
    if (unit < stride && (threadIdx.x < CK_NT / 64 || blockIdx.y == gridDim.y - 1))
        flags[row * stride + unit] = threadIdx.x >= CK_NT / 64 || !any_live[threadIdx.x] ? FL_DEAD
                                     : any_neg[threadIdx.x]                              ? FL_MIXED
                                                                                         : FL_CLEAN;
}

// states at the start of every CKR-l block (ck, with its flags per 64 pairs), and optionally at its
// quarter points l0 + CKR/4 (ck_q1), l0 + CKR/2 (ck_mid) and l0 + 3 CKR/4 (ck_q3), same indexing; a
// state past lmax is not written
__global__ void __launch_bounds__(CK_NT) ck_scalar_kernel(GeomDev g, int lmax, const int64_t *__restrict__ blk_ofs,
                                                          float4 *__restrict__ ck,
                                                          uint8_t *__restrict__ flags, float4 *__restrict__ ck_mid,
                                                          float4 *__restrict__ ck_q1 = nullptr,
                                                          float4 *__restrict__ ck_q3 = nullptr) {
    const int m = blockIdx.x;
    const int64_t p = (int64_t)blockIdx.y * CK_NT + threadIdx.x;
    __shared__ double2 cf[CKR];
    const int64_t np = g.npairs;
    const bool live = p < np;
    double x = live ? g.pair_x[p] : 0.0;
    double L = g.log2cm[m] + (double)m * (live ? g.pair_log2sin[p] : 0.0);
    int e = (int)floor((L + 256.0) / 512.0);
    double l1 = 0.0, l2 = exp2(L - 512.0 * e);
    if (m & 1) l2 = -l2;
    const int64_t o = blk_ofs[m] * np;
    __shared__ int any_neg[CK_NT / 64], any_live[CK_NT / 64];
    for (int l0 = m; l0 <= lmax; l0 += CKR) {
        const int64_t oj = o + (int64_t)((l0 - m) / CKR) * np + p;
        __syncthreads();
        for (int i = threadIdx.x; i < CKR; i += CK_NT) {
            int l = l0 + i;
            double A = 0.0, B = 1.0;
            if (l > m && l <= lmax) ck_scalar_coef(l, m, A, B);
            cf[i] = make_double2(A, B);
        }
        if (threadIdx.x < CK_NT / 64) any_neg[threadIdx.x] = any_live[threadIdx.x] = 0;
        __syncthreads();
        // state at the start of this block: (lambda_{l0-1}, lambda_{l0-2}); block 0 holds (0, lambda_mm)
        if (live && ck) {
            const float4 st = to_f32_state(l1, l2, e);
            ck[oj] = st;
            if (__float_as_int(st.z) < 0) any_neg[threadIdx.x / 64] = 1;
        }
        const int n = min(CKR, lmax - l0 + 1);
        for (int i = 0; i < n; ++i) {
            if (i == CKR / 2 && live && ck_mid) ck_mid[oj] = to_f32_state(l1, l2, e);
            if (i == CKR / 4 && live && ck_q1) ck_q1[oj] = to_f32_state(l1, l2, e);
            if (i == 3 * CKR / 4 && live && ck_q3) ck_q3[oj] = to_f32_state(l1, l2, e);
            double v = cf[i].x * x * l1 + cf[i].y * l2;
            l2 = l1;
            l1 = v;
            if (e < 0 && fabs(l1) > 0x1p256) {
                l1 *= 0x1p-512;
                l2 *= 0x1p-512;
                ++e;
            }
        }
        if (flags) {
            if (live && __float_as_int(to_f32_state(l1, l2, e).z) >= 0) any_live[threadIdx.x / 64] = 1;
            __syncthreads();
            write_flags(flags, blk_ofs[m] + (l0 - m) / CKR, np, any_neg, any_live);
        }
    }
}

// spin-2: P (s=+2 function, recursion with +b) and M (-b), blocks from l0 = max(m,2)
__device__ __forceinline__ void ck_spin_coef(int lp, int m, double &a, double &b, double &c) {
    const double l = lp - 1, mm = m;
    const double R1 = sqrt(((l + 1) * (l + 1) - mm * mm) * ((l + 1) * (l + 1) - 4.0));
    const double R0 = sqrt(fmax(0.0, (l * l - mm * mm) * (l * l - 4.0)));
    const double n10 = sqrt((2 * l + 3) / (2 * l + 1)), n1m = sqrt((2 * l + 3) / (2 * l - 1));
    a = n10 * (2 * l + 1) * (l + 1) / R1;
    b = n10 * (2 * l + 1) * 2.0 * mm / (l * R1);
    c = n1m * (l + 1) * R0 / (l * R1);
}

// (a, b, c) of the FP32 kernels, zero past lmax; l = max(m, 2) gives (0, 0, -1): the first block's
// state is (0, start value)
__global__ void spin32_coef_kernel(int lmax, const int64_t *__restrict__ blk_ofs, float4 *__restrict__ tab) {
    const int m = blockIdx.x, l0 = m > 2 ? m : 2;
    float4 *t = tab + blk_ofs[m] * CKR;
    const int64_t n = (blk_ofs[m + 1] - blk_ofs[m]) * CKR;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        double a = 0.0, b = 0.0, c = i == 0 ? -1.0 : 0.0;
        if (i > 0 && l0 + i <= lmax) ck_spin_coef(l0 + (int)i, m, a, b, c);
        t[i] = make_float4((float)a, (float)b, (float)c, 0.f);
    }
}

__global__ void __launch_bounds__(CK_NT) ck_spin_kernel(GeomDev g, int lmax, const int64_t *__restrict__ blk_ofs,
                                                        float4 *__restrict__ ckP, float4 *__restrict__ ckM,
                                                        uint8_t *__restrict__ flags) {
    const int m = blockIdx.x;
    const int64_t p = (int64_t)blockIdx.y * CK_NT + threadIdx.x;
    __shared__ double4 cf[CKR];
    const int64_t np = g.npairs;
    const bool live = p < np;
    const int l0s = m > 2 ? m : 2;
    double x = live ? g.pair_x[p] : 0.0;
    double lc = live ? g.pair_log2ch[p] : 0.0, ls = live ? g.pair_log2sh[p] : 0.0, k = g.log2spin[m];
    const int u = m + 2, v = m >= 2 ? m - 2 : 2 - m;
    double LP = k + v * lc + u * ls, LM = k + u * lc + v * ls;
    int ep = (int)floor((LP + 256.0) / 512.0), em = (int)floor((LM + 256.0) / 512.0);
    double sp = (m & 1) ? -1.0 : 1.0, sm = (m >= 2) ? sp : 1.0;
    double P1 = 0.0, P2 = sp * exp2(LP - 512.0 * ep), M1 = 0.0, M2 = sm * exp2(LM - 512.0 * em);
    float4 *oP = ckP + blk_ofs[m] * np, *oM = ckM + blk_ofs[m] * np;
    __shared__ int any_neg[CK_NT / 64], any_live[CK_NT / 64];
    for (int lb = l0s; lb <= lmax; lb += CKR) {
        __syncthreads();
        if (threadIdx.x < CK_NT / 64) any_neg[threadIdx.x] = any_live[threadIdx.x] = 0;
        __syncthreads();
        if (live) {
            const float4 sP = to_f32_state(P1, P2, ep), sM = to_f32_state(M1, M2, em);
            oP[(int64_t)((lb - l0s) / CKR) * np + p] = sP;
            oM[(int64_t)((lb - l0s) / CKR) * np + p] = sM;
            if (__float_as_int(sP.z) < 0 || __float_as_int(sM.z) < 0) any_neg[threadIdx.x / 64] = 1;
        }
        for (int i = threadIdx.x; i < CKR; i += CK_NT) {
            int lp = lb + i;
            double a = 0.0, b = 0.0, c = 0.0;
            if (lp == l0s) {
                c = -1.0;
            } else if (lp <= lmax) {
                ck_spin_coef(lp, m, a, b, c);
            }
            cf[i] = make_double4(a, b, c, 0.0);
        }
        __syncthreads();
        const int n = min(CKR, lmax - lb + 1);
        for (int i = 0; i < n; ++i) {
            const double4 q = cf[i];
            double vp = (q.x * x + q.y) * P1 - q.z * P2;
            double vm = (q.x * x - q.y) * M1 - q.z * M2;
            P2 = P1; P1 = vp; M2 = M1; M1 = vm;
            if (ep < 0 && fabs(P1) > 0x1p256) { P1 *= 0x1p-512; P2 *= 0x1p-512; ++ep; }
            if (em < 0 && fabs(M1) > 0x1p256) { M1 *= 0x1p-512; M2 *= 0x1p-512; ++em; }
        }
        if (live && (__float_as_int(to_f32_state(P1, P2, ep).z) >= 0 || __float_as_int(to_f32_state(M1, M2, em).z) >= 0))
            any_live[threadIdx.x / 64] = 1;
        __syncthreads();
        write_flags(flags, blk_ofs[m] + (lb - l0s) / CKR, np, any_neg, any_live);
    }
}

int launch_ck_mid(const hb_plan *p, float4 *ck_mid, float4 *ck_q1, float4 *ck_q3) {
    const int64_t np = p->g->d.npairs;
    dim3 grid((unsigned)(p->mmax + 1), (unsigned)((np + CK_NT - 1) / CK_NT));
    ck_scalar_kernel<<<grid, CK_NT>>>(p->g->d, p->lmax, p->blk_ofs, nullptr, nullptr, ck_mid, ck_q1, ck_q3);
    HB_CUDA_TRY(cudaGetLastError());
    return HB_OK;
}

}  // namespace hb

using namespace hb;

static int64_t nblk(int lmax, int lstart) { return lstart > lmax ? 0 : (lmax - lstart) / CKR + 1; }

extern "C" {

int hb_plan_create(const hb_geom *g, int lmax, int mmax, int flags, hb_plan **out) {
    if (!g || !out) return fail(HB_ERR_INVALID, "hb_plan_create: null argument");
    if (lmax < 0 || lmax > HB_MAX_L || mmax < 0 || mmax > lmax)
        return fail(HB_ERR_INVALID, "hb_plan_create: need 0 <= mmax <= lmax <= 16383");
    hb_plan *p = new hb_plan();
    p->g = g;
    p->lmax = lmax;
    p->mmax = mmax;
    p->flags = flags;
    const int64_t np = g->d.npairs;
    std::vector<int64_t> ofs(mmax + 2), ofs_s(mmax + 2), ofs_t(mmax + 2);
    ofs[0] = ofs_s[0] = ofs_t[0] = 0;
    for (int m = 0; m <= mmax; ++m) {
        ofs[m + 1] = ofs[m] + nblk(lmax, m);
        ofs_s[m + 1] = ofs_s[m] + nblk(lmax, m > 2 ? m : 2);
        ofs_t[m + 1] = ofs_t[m] + (lmax - m) / 2 + 1;
    }
    const bool scalar = (flags & HB_PLAN_FP32) != 0, spin = (flags & HB_PLAN_SPIN2_FP32) != 0, fp64 = !(flags & HB_PLAN_NO_FP64);
    size_t bytes = 0;
    auto carve = [&](size_t b) { size_t o = bytes; bytes += (b + 255) & ~(size_t)255; return o; };
    size_t o_ofs = carve(8 * (mmax + 2)), o_ofss = carve(8 * (mmax + 2)), o_ofst = carve(8 * (mmax + 2));
    const size_t o_leg = fp64 ? carve(8 * LT_N * (size_t)ofs_t[mmax + 1]) : 0;
    const size_t o_flags = scalar ? carve((size_t)ofs[mmax + 1] * flag_stride(np)) : 0;
    const size_t o_leg32 = scalar ? carve(8 * (size_t)ofs[mmax + 1] * CKR) : 0;
    size_t o_ck = scalar ? carve(16 * (size_t)ofs[mmax + 1] * np) : 0;
    const size_t o_spin32 = spin ? carve(16 * (size_t)ofs_s[mmax + 1] * CKR) : 0;
    const size_t o_flags_s = spin ? carve((size_t)ofs_s[mmax + 1] * flag_stride(np)) : 0;
    size_t o_ckp = spin ? carve(16 * (size_t)ofs_s[mmax + 1] * np) : 0;
    size_t o_ckm = spin ? carve(16 * (size_t)ofs_s[mmax + 1] * np) : 0;
    char *base = nullptr;
    if (cudaMalloc(&base, bytes) != cudaSuccess) {
        cudaGetLastError();
        delete p;
        return fail(HB_ERR_ALLOC, "hb_plan_create: cudaMalloc of " + std::to_string(bytes) + " bytes failed");
    }
    p->alloc_base = base;
    p->bytes = bytes;
    p->blk_ofs = (int64_t *)(base + o_ofs);
    p->blk_ofs_spin = (int64_t *)(base + o_ofss);
    p->leg = {fp64 ? (double *)(base + o_leg) : nullptr, (int64_t *)(base + o_ofst)};
    p->leg32 = scalar ? (float2 *)(base + o_leg32) : nullptr;
    p->ck_flags = scalar ? (uint8_t *)(base + o_flags) : nullptr;
    p->ck = scalar ? (float4 *)(base + o_ck) : nullptr;
    p->spin32 = spin ? (float4 *)(base + o_spin32) : nullptr;
    p->ck_flags_spin = spin ? (uint8_t *)(base + o_flags_s) : nullptr;
    p->ckP = spin ? (float4 *)(base + o_ckp) : nullptr;
    p->ckM = spin ? (float4 *)(base + o_ckm) : nullptr;
    int rc = HB_OK;
    if (cudaMemcpy(p->blk_ofs, ofs.data(), 8 * (mmax + 2), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(p->blk_ofs_spin, ofs_s.data(), 8 * (mmax + 2), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(p->leg.ofs, ofs_t.data(), 8 * (mmax + 2), cudaMemcpyHostToDevice) != cudaSuccess)
        rc = fail(HB_ERR_CUDA, "hb_plan_create: upload failed");
    dim3 grid((unsigned)(mmax + 1), (unsigned)((np + CK_NT - 1) / CK_NT));
    if (rc == HB_OK) {
        if (fp64) leg_table_kernel<<<(unsigned)(mmax / 32 + 1), 32>>>(lmax, mmax, p->leg);
        if (scalar) leg32_coef_kernel<<<(unsigned)(mmax + 1), 256>>>(lmax, p->blk_ofs, p->leg32);
        if (cudaGetLastError() != cudaSuccess) rc = fail(HB_ERR_CUDA, "hb_plan_create: table kernel launch");
    }
    if (rc == HB_OK && scalar) {
        ck_scalar_kernel<<<grid, CK_NT>>>(g->d, lmax, p->blk_ofs, p->ck, p->ck_flags, nullptr);
        if (cudaGetLastError() != cudaSuccess) rc = fail(HB_ERR_CUDA, "hb_plan_create: checkpoint kernel launch");
    }
    if (rc == HB_OK && spin) {
        spin32_coef_kernel<<<(unsigned)(mmax + 1), 256>>>(lmax, p->blk_ofs_spin, p->spin32);
        ck_spin_kernel<<<grid, CK_NT>>>(g->d, lmax, p->blk_ofs_spin, p->ckP, p->ckM, p->ck_flags_spin);
        if (cudaGetLastError() != cudaSuccess) rc = fail(HB_ERR_CUDA, "hb_plan_create: spin checkpoint kernel launch");
    }
    if (rc == HB_OK && cudaDeviceSynchronize() != cudaSuccess) rc = fail(HB_ERR_CUDA, "hb_plan_create: table build failed");
    if (rc != HB_OK) {
        cudaFree(base);
        delete p;
        return rc;
    }
    *out = p;
    return HB_OK;
}

int hb_plan_destroy(hb_plan *p) {
    if (!p) return HB_OK;
    cudaFree(p->alloc_base);
    delete p;
    return HB_OK;
}

size_t hb_plan_bytes(const hb_plan *p) { return p ? p->bytes : 0; }

}  // extern "C"
