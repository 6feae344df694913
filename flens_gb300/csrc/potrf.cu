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
// trsm); on the GPU, by blocks of 256 columns,
//
//   factor A11;  A21 <- A21 L11^-T  (trsm);  A22 -= A21 A21^T  (syrk, lower tiles only)
//
// with the 256-deep updates on the tensor cores (mod_gemm.cu), the next diagonal
// block first, which is then factored beside the rest; a diagonal block takes the
// same three steps 64 columns at a time with potf2 of the 64 x 64 block in one CTA.
// n = 4000 with one right-hand side: 31.6 ms with right-looking 64-column steps on
// the FP64 pipe, 11.1 one after the other, 8.3 in this order.
//
// Pivots, INFO and the factor agree with the reference to rounding; when
// INFO > 0 the columns from the failing 64-column step on hold the updates of all
// whole steps before it and nothing else but the columns of its own 64 x 64 block
// before the pivot (the reference leaves them as they were, LAPACK undefined).
#include "common.cuh"

#include <math_constants.h>

#include <cmath>

namespace fg {

namespace {

constexpr int POTRF_NB = 64;
constexpr int POTRF_BASE = 256;
constexpr int kSideSms = 16;                      // left to the side stream

// Unblocked right-looking Cholesky of the jb x jb (jb <= 64) diagonal block
// at A, whose lower-view element (i, c), i >= c, is A[i*rs + c*cs] (rs = 1,
// cs = ld for 'L'; rs = ld, cs = 1 for 'U').  On a pivot <= 0 or NaN in
// column f it stores that pivot, writes back columns < f only and sets
// *info = j0 + f + 1.  Does nothing when *info is already set.
//
// Bound: the chain of the pivots and the FP64 pipe behind it (a dependent FP64
// instruction takes about 100 clocks, a warp's instruction 16 of the SM's pipe).  The
// elimination therefore runs on the unscaled columns, a_ic -= (a_it p_t) a_ct with
// p_t = 1 / pivot, in three stages beside each other, one barrier per step t:
//   warp 0        column t + 1 (the half that holds its pivot) with column t, as
//                 (a_it a_ct) p_t: the product is formed while the reciprocal before
//                 is under way, so that one FMA and a reciprocal stand on the chain;
//                 warp 3 its other half;
//   warps 1, 2    column t + 2 with columns t - 1 and t;
//   the other 8   column t - 1 to the columns from t + 3 on, which they hold in
//                 registers in 8 x 4 tiles and store as each becomes column t + 3.
// The columns are scaled by 1 / sqrt(pivot) and the diagonal's square roots taken at
// the end, together.  A block takes 43 us: 4 of launch, load and store, 9 of
// divisions.  93 with sqrt, divide and three barriers per column on the chain; 57 with
// the trailing block in shared memory, whose masked lanes took 2560 warp FMAs instead
// of 1500, and two FMAs and a multiplication on the chain.  More warps only lengthen
// the barriers (512 threads: 45).
constexpr int POTF2_THREADS = 384, UPD = POTF2_THREADS / 32 - 4;
constexpr int TILES = 72, UPD_TILES = (TILES + UPD - 1) / UPD;      // 8 x 4 tiles that meet the triangle

// The block with each column scaled by 1 / sqrt(pivot) as it is reached, so that no
// product exceeds the square root of two diagonal entries: for pivots beyond 2^+-250,
// and where the elimination above left an infinity or NaN.  (Between pivots in that
// range a reciprocal is a normal number, but the unscaled product a_it a_ct of a large
// row still overflows: [2^200 2^600; 2^600 2^1001]; and one of two entries below 2^-480
// may lose bits that the reciprocal of a pivot below 2^-50 brings back into range.)  Returns the failing column + 1,
// or 0.
__device__ __noinline__ int potf2_plain(double (*S)[POTRF_NB + 1], int jb, const double *A, size_t rs, size_t cs) {
    const int tid = threadIdx.x;
    __syncthreads();
    for (int e = tid; e < POTRF_NB * POTRF_NB; e += POTF2_THREADS) {
        const int i = e % POTRF_NB, c = e / POTRF_NB;
        S[c][i] = (i >= c && i < jb) ? A[(size_t)i * rs + (size_t)c * cs] : 0.0;
    }
    __syncthreads();
    for (int t = 0; t < jb; ++t) {
        const double a = S[t][t];
        if (!(a > 0.0)) return t + 1;
        const double d = sqrt(a), r = 1.0 / d;
        __syncthreads();
        if (tid >= t && tid < POTRF_NB) S[t][tid] = tid > t ? S[t][tid] * r : d;
        __syncthreads();
        for (int e = tid; e < POTRF_NB * POTRF_NB; e += POTF2_THREADS) {
            const int i = e % POTRF_NB, c = e / POTRF_NB;
            if (c > t && i >= c) S[c][i] = fma(-S[t][i], S[t][c], S[c][i]);
        }
        __syncthreads();
    }
    return 0;
}

__global__ void __launch_bounds__(POTF2_THREADS)
potf2_kernel(int jb, double *__restrict__ A, size_t rs, size_t cs, int j0, int *__restrict__ info) {
    __shared__ double S[POTRF_NB][POTRF_NB + 1];      // S[c][i] = element (i, c), unscaled
    __shared__ double Lp[2][POTRF_NB];                // column t times p_t
    __shared__ double s_p[POTRF_NB];                  // 1 / pivot, later 1 / sqrt(pivot)
    __shared__ int s_fail, s_skip, s_odd;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_fail = 0;
        s_skip = *info != 0;
        s_odd = 0;
    }
#pragma unroll
    for (int h = 0; h < (POTRF_NB * POTRF_NB + POTF2_THREADS - 1) / POTF2_THREADS; ++h) {
        const int e = h * POTF2_THREADS + tid, lo = e % POTRF_NB, hi = e / POTRF_NB;
        if (hi >= POTRF_NB) break;
        const int i = rs == 1 ? lo : hi, c = rs == 1 ? hi : lo;
        S[c][i] = (i >= c && i < jb) ? A[(size_t)i * rs + (size_t)c * cs] : 0.0;
    }
    __syncthreads();
    if (s_skip) return;
    // Warp 0's: p = 1 / pivot of column t, w = column t times its row t + 1
    double p = 0.0, w = 0.0;
    auto pivot = [&](double a, int j) {               // by warp 0
        // in [2^-250, 2^251), by its exponent and sign
        if ((unsigned)((__double_as_longlong(a) >> 52) & 0xFFF) - 773u > 500u) {
            if (lane == 0) s_fail = j + 1;
        } else {
            p = 1.0 / a;
            if (lane == 0) s_p[j] = p;
        }
    };
    // the updating warps' tiles: 8 rows x 4 columns, the last columns first, so that
    // the tiles still open in a step are the first of the list
    double v[UPD_TILES];
    int ti[UPD_TILES], tc[UPD_TILES];
    if (warp >= 4) {
#pragma unroll
        for (int h = 0; h < UPD_TILES; ++h) {
            const int idx = warp - 4 + UPD * h;
            int q = 0;
            while ((q + 1) * (q + 2) <= idx) ++q;
            const int r = idx - q * (q + 1), far = r > q;
            ti[h] = 8 * (7 - (far ? r - q - 1 : r)) + (lane & 7);
            tc[h] = 4 * (15 - 2 * q - far) + (lane >> 3);
            v[h] = idx < TILES ? S[tc[h]][ti[h]] : 0.0;
        }
    } else if (warp == 0) {
        pivot(S[0][0], 0);
    }
    __syncthreads();
    int fail = 0;
    for (int t = 0; t < jb; ++t) {
        // (a warp may see the failure of pivot t + 1, found in this step: not yet)
        fail = s_fail == t + 1 ? t + 1 : 0;
        if (fail) break;
        if (warp == 0) {
            if (t + 1 < jb) {
                const int i = lane + (t + 1 < 32 ? 0 : 32);
                if (t == 0 || t == 31) w = S[t][i] * S[t][t + 1];      // (rows 32 .. 63 from t = 31 on)
                const double x = fma(-w, p, S[t + 1][i]);
                pivot(__shfl_sync(0xffffffffu, x, (t + 1) & 31), t + 1);
                if (i > t) S[t + 1][i] = x;
                w = x * __shfl_sync(0xffffffffu, x, (t + 2) & 31);
            }
        } else if (warp == 3) {
            if (t + 1 < 32) {
                const int i = lane + 32;
                S[t + 1][i] = fma(-(S[t][i] * s_p[t]), S[t][t + 1], S[t + 1][i]);
            }
        } else if (warp < 3) {
            const int i = lane + 32 * (warp - 1);
            const double l = S[t][i] * s_p[t];
            Lp[t & 1][i] = l;
            if (i >= t + 2) {
                double y = S[t + 2][i];
                if (t > 0) y = fma(-Lp[(t - 1) & 1][i], S[t - 1][t + 2], y);
                S[t + 2][i] = fma(-l, S[t][t + 2], y);
            }
        } else if (t > 0) {
            const int k = 16 - ((t + 3) >> 2), q = k >> 1, open = q * (q + 1) + (k & 1) * (q + 1);
#pragma unroll
            for (int h = 0; h < UPD_TILES; ++h) {
                if (warp - 4 + UPD * h >= open) break;
                v[h] = fma(-Lp[(t - 1) & 1][ti[h]], S[t - 1][tc[h]], v[h]);
                if (tc[h] == t + 3 && ti[h] >= t + 3) S[t + 3][ti[h]] = v[h];
            }
        }
        __syncthreads();
    }
    // The block starts again after a positive pivot beyond the range (bit 0), an overflow,
    // which stays where it arose: as an infinity or NaN in a column to be stored,
    // -infinity on the diagonal (a NaN there alone was in A), and where bits may be lost:
    // an entry below 2^-480 (bit 1) and a pivot below 2^-50 (bit 2).  High words only, and
    // beside the roots, which the diagonal's threads take.
    int ncol = fail ? fail - 1 : jb;
    unsigned odd = fail && (S[fail - 1][fail - 1] > 0.0 || S[fail - 1][fail - 1] == -CUDART_INF) ? 1u : 0u;
    unsigned most = 0u, least = ~0u;                  // of |entry|, least: of the nonzeros, less one
#pragma unroll
    for (int h = 0; h < (POTRF_NB * POTRF_NB + POTF2_THREADS - 1) / POTF2_THREADS; ++h) {
        const int e = h * POTF2_THREADS + tid, i = e % POTRF_NB, c = e / POTRF_NB;
        const unsigned u = i > c && c < ncol ? (unsigned)__double2hiint(S[c][i]) & 0x7FFFFFFFu : 0u;
        most = max(most, u);
        least = min(least, u - 1u);
    }
    if (tid < ncol) {
        const double a = S[tid][tid];
        const unsigned u = (unsigned)__double2hiint(a);
        most = max(most, u);
        if (u < (1023u - 50u) << 20) odd |= 4u;
        S[tid][tid] = sqrt(a);
        s_p[tid] = rsqrt(a);
    }
    odd |= (most >= 0x7FFu << 20 ? 1u : 0u) | (least < (1023u - 480u) << 20 ? 2u : 0u);
    odd = __reduce_or_sync(0xffffffffu, odd);
    if (odd && lane == 0) atomicOr(&s_odd, (int)odd);
    __syncthreads();
    if ((s_odd & 1) || (s_odd & 6) == 6) {
        fail = potf2_plain(S, jb, A, rs, cs);
        ncol = fail ? fail - 1 : jb;
        if (tid < POTRF_NB) s_p[tid] = 1.0;
        __syncthreads();
    }
#pragma unroll
    for (int h = 0; h < (POTRF_NB * POTRF_NB + POTF2_THREADS - 1) / POTF2_THREADS; ++h) {
        const int e = h * POTF2_THREADS + tid, lo = e % POTRF_NB, hi = e / POTRF_NB;
        if (hi >= POTRF_NB) break;
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
    auto at = [&](int i, int j) { return lower ? A + i + (size_t)j * ldA : A + j + (size_t)i * ldA; };   // element (i, j) of L
    // Of a factored block of width w at j: rows r0 .. r0 + nr - 1 of L below it ...
    auto solve_rows = [&](int j, int w, int r0, int nr, cudaStream_t q) -> int {
        return lower ? dtrsm_launch('R', 'L', 'T', 'N', nr, w, 1.0, at(j, j), ldA, at(r0, j), ldA, q)
                     : dtrsm_launch('L', 'U', 'T', 'N', w, nr, 1.0, at(j, j), ldA, at(r0, j), ldA, q);
    };
    // ... their update of the triangle at c0, nc wide, and of the rows r0 .. below it
    auto update_diag = [&](int j, int w, int c0, int nc, cudaStream_t q) -> int {
        return dsyrk_launch(lower ? 'L' : 'U', lower ? 'N' : 'T', nc, w, -1.0, at(c0, j), ldA, 1.0, at(c0, c0), ldA, q);
    };
    auto update_below = [&](int j, int w, int c0, int nc, int r0, int nr, cudaStream_t q) -> int {
        return lower ? dgemm_launch('N', 'T', nr, nc, w, -1.0, at(r0, j), ldA, at(c0, j), ldA, 1.0, at(r0, c0), ldA, q)
                     : dgemm_launch('T', 'N', nc, nr, w, -1.0, at(c0, j), ldA, at(r0, j), ldA, 1.0, at(r0, c0), ldA, q);
    };
    // A diagonal block of up to POTRF_BASE columns, right-looking in steps of 64.  After
    // a failed pivot its step's solve and update, and the steps behind it, leave the
    // matrix as it is (by *info, on the device).
    auto diagonal = [&](int j, int w, cudaStream_t q) -> int {
        for (int c = 0; c < w; c += POTRF_NB) {
            const int jb = w - c < POTRF_NB ? w - c : POTRF_NB, rest = w - c - jb;
            {
                KTimer kt(kFamPanel, q, (double)jb * jb * jb / 3.0, 16.0 * jb * jb);
                potf2_kernel<<<1, POTF2_THREADS, 0, q>>>(jb, at(j + c, j + c), rs, cs, j + c, info);
                FG_CUDA(cudaGetLastError());
            }
            if (rest <= 0) break;
            const int c0 = j + c, r0 = c0 + jb;
            int st = lower ? dtrsm_block_launch('R', 'L', 'T', 'N', rest, jb, 1.0, at(c0, c0), ldA, at(r0, c0), ldA, info, q)
                           : dtrsm_block_launch('L', 'U', 'T', 'N', jb, rest, 1.0, at(c0, c0), ldA, at(r0, c0), ldA, info, q);
            if (st != kOk) return st;
            if ((st = dsyrk_launch(lower ? 'L' : 'U', lower ? 'N' : 'T', rest, jb, -1.0, at(r0, c0), ldA, 1.0,
                                   at(r0, r0), ldA, q, info)) != kOk)
                return st;
        }
        return kOk;
    };
    // The block of width w at j failed in column f: what its whole 64-column steps
    // before f mean for the rows below it and the columns behind them, so that the
    // matrix is left as if the step of f had been the first not taken.
    auto finish = [&](int j, int w, int f) -> int {
        const int w0 = (f - j) / POTRF_NB * POTRF_NB, e = j + w, c0 = j + w0;
        if (w0 == 0 || e == n) return kOk;
        int st = solve_rows(j, w0, e, n - e, s);
        if (st == kOk) st = update_below(j, w0, c0, e - c0, e, n - e, s);
        if (st == kOk) st = update_diag(j, w0, e, n - e, s);
        return st;
    };
    if (n <= 2 * POTRF_BASE) {
        // few blocks: one after the other; INFO is read back after each but the last
        for (int j = 0; j < n; j += POTRF_BASE) {
            const int w = n - j < POTRF_BASE ? n - j : POTRF_BASE, rest = n - j - w;
            int st = diagonal(j, w, s);
            if (st != kOk || rest == 0) return st;
            FG_CUDA(cudaMemcpyAsync(h, info, sizeof(int), cudaMemcpyDeviceToHost, s));
            FG_CUDA(cudaStreamSynchronize(s));
            if (*h != 0) return finish(j, w, *h - 1);           // as potrf.tcc:104-107 stops
            if ((st = solve_rows(j, w, j + w, rest, s)) != kOk) return st;
            if ((st = update_diag(j, w, j + w, rest, s)) != kOk) return st;
        }
        return kOk;
    }
    // Look-ahead: a diagonal block is a chain of small launches (240 us for 256
    // columns), so the next one is updated first and factored on the side stream
    // while the rest of the update, whose persistent products leave it 16 SMs, runs
    // here.  n = 4000 with one right-hand side: 11.1 ms without.
    Workspace *wo = workspace_side(s);
    if (!wo) return kErrCuda;
    cudaStream_t side = wo->side;
    bool open = false;                            // side-stream work not yet joined
    auto start = [&](int j, int w) -> int {       // diagonal block and its INFO, after what s has
        FG_CUDA(cudaEventRecord(wo->ev_fwd, s));
        FG_CUDA(cudaStreamWaitEvent(side, wo->ev_fwd, 0));
        open = true;
        const int st = diagonal(j, w, side);
        // (not after the last block: a copy in flight when the call returns could land
        // in a later call's readback)
        if (st == kOk && j + w < n) FG_CUDA(cudaMemcpyAsync(h, info, sizeof(int), cudaMemcpyDeviceToHost, side));
        FG_CUDA(cudaEventRecord(wo->ev_back, side));
        return st;
    };
    auto run = [&]() -> int {
        int st = start(0, POTRF_BASE);
        for (int j = 0, w = POTRF_BASE; st == kOk;) {
            const int e = j + w;
            FG_CUDA(cudaStreamWaitEvent(s, wo->ev_back, 0));
            open = false;
            if (e == n) break;
            FG_CUDA(cudaEventSynchronize(wo->ev_back));
            if (*h != 0) return finish(j, w, *h - 1);           // as potrf.tcc:104-107 stops
            const int w2 = n - e < POTRF_BASE ? n - e : POTRF_BASE, e2 = e + w2;
            if ((st = solve_rows(j, w, e, w2, s)) != kOk) return st;
            if ((st = update_diag(j, w, e, w2, s)) != kOk) return st;
            if ((st = start(e, w2)) != kOk) return st;
            if (n > e2) {
                SpareSms spare(kSideSms);
                if ((st = solve_rows(j, w, e2, n - e2, s)) != kOk) return st;
                if ((st = update_below(j, w, e, w2, e2, n - e2, s)) != kOk) return st;
                if ((st = update_diag(j, w, e2, n - e2, s)) != kOk) return st;
            }
            j = e;
            w = w2;
        }
        return st;
    };
    const int st = run();
    // never leave side-stream work unjoined, also on an error path
    if (open) cudaStreamWaitEvent(s, wo->ev_back, 0);
    if (st != kOk) {
        cudaStreamSynchronize(side);              // its readback, too
        return st;
    }
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
