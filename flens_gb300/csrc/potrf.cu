// potrf.cu -- Cholesky factorisation and solve, FP64, column-major.
//
//   dpotrf: A = L L^T (uplo 'L') or U^T U ('U') in place, the other triangle
//           untouched; INFO = first column whose pivot is <= 0 or NaN.
//   dpotrs: A X = B from the factor (two triangular solves).
//
// Follows FLENS-LAPACK potrf (flens/lapack/po/potrf.tcc:56-150, block size 64
// from ilaenv PO/TRF, flens/lapack/la/ilaenv.tcc:126-132), potf2
// (flens/lapack/po/potf2.tcc:56-140: pivot test `ajj <= 0 || isnan(ajj)`,
// the failing pivot stored in A(j,j), column scaled by the reciprocal 1/ajj)
// and potrs (flens/lapack/po/potrs.tcc:54-100).  The reference updates
// left-looking (syrk of the diagonal block, gemm of the block column, then
// trsm); on the GPU the columns are halved down to 256,
//
//   factor(left half);  A21 <- A21 L11^-T  (trsm);  A22 -= A21 A21^T  (syrk, lower
//   tiles only);  factor(right half)
//
// so that the updates are deep products, and a block of 256 columns takes the
// same three steps 64 columns at a time with potf2 of the 64 x 64 diagonal block
// in one CTA.  n = 4000 with one right-hand side: 31.6 ms with right-looking
// 64-column steps on the FP64 pipe, 17.5 with their products on the tensor cores,
// 11.5 halved and with the diagonal block below.
//
// Pivots, INFO and the factor agree with the reference to rounding; when
// INFO > 0 the columns after the failing block hold partially updated values
// (the reference leaves them as they were), as LAPACK leaves them undefined.
#include "common.cuh"

#include <cmath>

namespace fg {

namespace {

constexpr int POTRF_NB = 64;
constexpr int POTRF_BASE = 256;

// Unblocked right-looking Cholesky of the jb x jb (jb <= 64) diagonal block
// at A, whose lower-view element (i, c), i >= c, is A[i*rs + c*cs] (rs = 1,
// cs = ld for 'L'; rs = ld, cs = 1 for 'U').  On a pivot <= 0 or NaN in
// column f it stores that pivot, writes back columns < f only and sets
// *info = j0 + f + 1.  Does nothing when *info is already set.
//
// Bound: the chain of the pivots, as one FP64 instruction holds a scheduler's
// pipe for 64 clocks and takes about 100.  The elimination therefore runs on the
// unscaled columns, a_ic -= (a_it p_t) a_ct with p_t = 1 / pivot: two FP64
// instructions and a reciprocal (three, see recip) per step.  Warps 0 and 1
// (thread per row) run that chain: in step t they bring column t + 1 up to date
// with columns t - 1 and t, and the warp that owns the next pivot takes its
// reciprocal.  The other 14 apply column t - 1 to the columns from t + 2 on, one
// barrier per step.  The columns are scaled by 1 / sqrt(pivot) and the diagonal's
// square roots taken at the end, together.  (With sqrt, divide and three barriers
// per column on the chain a block took 93 us; this takes 55.)
constexpr int POTF2_THREADS = 512, UPD = POTF2_THREADS / 32 - 2;

// 1 / d for a normal d within 2^+-1000, to about an ulp: the FP32 reciprocal r of
// its significand, then the third-order iteration r + r (e + e^2), e = 1 - d r.
__device__ __forceinline__ double recip(double d) {
    const long long b = __double_as_longlong(d);
    const int ex = (int)(b >> 52) & 0x7FF;
    if (ex < 23 || ex > 2023) return 1.0 / d;
    // significand in [1, 2) as FP32 (its leading 23 bits), and d scaled to it
    const float f = __uint_as_float(0x3F800000u | (unsigned)((b >> 29) & 0x7FFFFF));
    const unsigned r = __float_as_uint(__fdividef(1.0f, f));           // in [0.5, 1]
    const double m = __longlong_as_double((b & 0xFFFFFFFFFFFFFll) | 0x3FF0000000000000ll);
    const double x = __longlong_as_double(((long long)((r >> 23) + 896) << 52) | ((long long)(r & 0x7FFFFFu) << 29));
    const double e = fma(-m, x, 1.0);
    const double y = fma(x, fma(e, e, e), x);
    return __longlong_as_double(__double_as_longlong(y) - ((long long)(ex - 1023) << 52));
}

__global__ void __launch_bounds__(POTF2_THREADS)
potf2_kernel(int jb, double *__restrict__ A, size_t rs, size_t cs, int j0, int *__restrict__ info) {
    __shared__ double S[POTRF_NB][POTRF_NB + 1];      // S[c][i] = element (i, c), unscaled
    __shared__ double Lp[2][POTRF_NB];                // column t times p_t
    __shared__ double s_p[POTRF_NB];                  // 1 / pivot, later 1 / sqrt(pivot)
    __shared__ int s_fail, s_skip;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_fail = 0;
        s_skip = *info != 0;
    }
#pragma unroll
    for (int h = 0; h < POTRF_NB * POTRF_NB / POTF2_THREADS; ++h) {
        const int e = h * POTF2_THREADS + tid, lo = e % POTRF_NB, hi = e / POTRF_NB;
        const int i = rs == 1 ? lo : hi, c = rs == 1 ? hi : lo;
        S[c][i] = (i >= c && i < jb) ? A[(size_t)i * rs + (size_t)c * cs] : 0.0;
    }
    __syncthreads();
    if (s_skip) return;
    auto pivot = [&](double a, int j) {               // by a whole warp
        const long long b = __double_as_longlong(a);
        if (b <= 0 || b > 0x7FF0000000000000ll) {     // a <= 0 or NaN
            if (lane == 0) s_fail = j + 1;
        } else {
            const double p = recip(a);
            if (lane == 0) s_p[j] = p;
        }
    };
    if (warp == 0) pivot(S[0][0], 0);
    __syncthreads();
    int fail = 0;
    for (int t = 0; t < jb; ++t) {
        fail = s_fail;
        if (fail) break;
        if (warp < 2) {
            const int i = tid;
            if (t + 1 < jb) {
                const double at = S[t][t + 1];
                double v = S[t + 1][i];
                if (t > 0) v = fma(-Lp[(t - 1) & 1][i], S[t - 1][t + 1], v);
                const double l = S[t][i] * s_p[t];
                v = fma(-l, at, v);
                if (((t + 1) >> 5) == warp) pivot(__shfl_sync(0xffffffffu, v, (t + 1) & 31), t + 1);
                Lp[t & 1][i] = l;
                if (i > t) S[t + 1][i] = v;
            }
        } else if (t > 0) {
            // units (column, row half) round robin over the other warps, four in
            // flight: the loads do not wait for the stores before them
            const int n1 = POTRF_NB - t - 2, n = n1 + (t + 2 < 32 ? 30 - t : 0);
            const double l0 = Lp[(t - 1) & 1][lane], l1 = Lp[(t - 1) & 1][lane + 32];
            for (int u = warp - 2; u < n; u += 4 * UPD) {
                double *e[4], v[4], a[4];
                bool in[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int w = u + UPD * h, lo = w >= n1, c = t + 2 + (lo ? w - n1 : w), i = (lo ? 0 : 32) + lane;
                    in[h] = w < n && i >= c;
                    e[h] = &S[in[h] ? c : 0][in[h] ? i : 0];
                    a[h] = in[h] ? S[t - 1][c] : 0.0;
                    v[h] = *e[h];
                }
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    if (u + UPD * h >= n) break;
                    v[h] = fma(-(u + UPD * h >= n1 ? l0 : l1), a[h], v[h]);
                    if (in[h]) *e[h] = v[h];
                }
            }
        }
        __syncthreads();
    }
    const int ncol = fail ? fail - 1 : jb;
    if (tid < ncol) {
        const double a = S[tid][tid];
        S[tid][tid] = sqrt(a);
        s_p[tid] = rsqrt(a);
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < POTRF_NB * POTRF_NB / POTF2_THREADS; ++h) {
        const int e = h * POTF2_THREADS + tid, lo = e % POTRF_NB, hi = e / POTRF_NB;
        const int i = rs == 1 ? lo : hi, c = rs == 1 ? hi : lo;
        if (i >= c && i < jb && c < ncol)
            A[(size_t)i * rs + (size_t)c * cs] = i > c ? S[c][i] * s_p[c] : S[c][i];
    }
    if (fail && tid == 0) {
        const int f = fail - 1;
        A[(size_t)f * (rs + cs)] = S[f][f];
        *info = j0 + fail;
    }
}

int *pinned_info() {
    thread_local int *h = nullptr;
    if (!h && cudaMallocHost((void **)&h, sizeof(int)) != cudaSuccess) {
        cudaGetLastError();
        h = nullptr;
    }
    return h;
}

}  // namespace

int dpotrf_launch(char uplo, int n, double *A, int ldA, int *info, cudaStream_t s) {
    FG_CUDA(cudaMemsetAsync(info, 0, sizeof(int), s));
    if (n == 0) return kOk;
    const bool lower = uplo == 'L' || uplo == 'l';
    const size_t rs = lower ? 1 : (size_t)ldA, cs = lower ? (size_t)ldA : 1;
    int *h = pinned_info();
    if (!h) {
        set_last_error("cudaMallocHost of the INFO readback failed");
        return kErrAlloc;
    }
    // rows below (lower) or columns right of (upper) a factored block of width w at
    // j, `rest` of them, and their update of what follows
    auto trailing = [&](int j, int w, int rest) -> int {
        double *A11 = A + j + (size_t)j * ldA, *A22 = A11 + w + (size_t)w * ldA;
        int st;
        if (lower) {
            double *A21 = A11 + w;
            if ((st = dtrsm_launch('R', 'L', 'T', 'N', rest, w, 1.0, A11, ldA, A21, ldA, s)) != kOk) return st;
            return dsyrk_launch('L', 'N', rest, w, -1.0, A21, ldA, 1.0, A22, ldA, s);
        }
        double *A12 = A11 + (size_t)w * ldA;
        if ((st = dtrsm_launch('L', 'U', 'T', 'N', w, rest, 1.0, A11, ldA, A12, ldA, s)) != kOk) return st;
        return dsyrk_launch('U', 'T', rest, w, -1.0, A12, ldA, 1.0, A22, ldA, s);
    };
    // Halved down to blocks of POTRF_BASE columns, so that the updates are as deep
    // as wide (tensor cores, mod_gemm.cu); those blocks go right-looking in steps
    // of 64.  *failed: a pivot failed (read back once per base block, as
    // potrf.tcc:104-107 stops there; inside a base block the remaining steps skip).
    auto factor = [&](auto &&self, int j, int w, bool last, bool *failed) -> int {
        int st;
        if (w > POTRF_BASE) {
            const int h = ceil_div(ceil_div(w, 2), POTRF_NB) * POTRF_NB;
            if ((st = self(self, j, h, false, failed)) != kOk || *failed) return st;
            if ((st = trailing(j, h, w - h)) != kOk) return st;
            return self(self, j + h, w - h, last, failed);
        }
        for (int c = 0; c < w; c += POTRF_NB) {
            const int jb = w - c < POTRF_NB ? w - c : POTRF_NB;
            {
                KTimer kt(kFamPanel, s, (double)jb * jb * jb / 3.0, 16.0 * jb * jb);
                potf2_kernel<<<1, POTF2_THREADS, 0, s>>>(jb, A + (j + c) + (size_t)(j + c) * ldA, rs, cs, j + c, info);
                FG_CUDA(cudaGetLastError());
            }
            if (c + jb < w && (st = trailing(j + c, jb, w - c - jb)) != kOk) return st;
        }
        if (last) return kOk;
        FG_CUDA(cudaMemcpyAsync(h, info, sizeof(int), cudaMemcpyDeviceToHost, s));
        FG_CUDA(cudaStreamSynchronize(s));
        *failed = *h != 0;
        return kOk;
    };
    bool failed = false;
    const int st = factor(factor, 0, n, true, &failed);
    if (st != kOk) return st;
    trace("potrf %c n=%d", uplo, n);
    return kOk;
}

// flens/lapack/po/potrs.tcc:54-100: L X = B then L^T X = B (lower), or
// U^T X = B then U X = B (upper).
int dpotrs_launch(char uplo, int n, int nrhs, const double *A, int ldA, double *B, int ldB,
                  cudaStream_t s) {
    if (n == 0 || nrhs == 0) return kOk;
    const bool lower = uplo == 'L' || uplo == 'l';
    int st;
    if (lower) {
        if ((st = dtrsm_launch('L', 'L', 'N', 'N', n, nrhs, 1.0, A, ldA, B, ldB, s)) != kOk) return st;
        return dtrsm_launch('L', 'L', 'T', 'N', n, nrhs, 1.0, A, ldA, B, ldB, s);
    }
    if ((st = dtrsm_launch('L', 'U', 'T', 'N', n, nrhs, 1.0, A, ldA, B, ldB, s)) != kOk) return st;
    return dtrsm_launch('L', 'U', 'N', 'N', n, nrhs, 1.0, A, ldA, B, ldB, s);
}

}  // namespace fg
