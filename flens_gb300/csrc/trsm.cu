// trsm.cu -- FP64 triangular solve with many right-hand sides.
//
// Replaces cxxblas::trsm for double (cxxblas/level3/trsm.tcc:40-82, reached
// from flens::blas::sm flens/blas/level3/sm.tcc:42-72 and dtrsm_
// flens/blas/interface/blas/trsm.cc:90-166).  As in the reference, alpha is
// applied AFTER the solve (trsm.tcc:67).
//
// All eight side/uplo/trans variants reduce to one description: an effective
// triangle M (op(A) for side=Left, op(A)^T for side=Right) addressed as
// M(i,p) = A[i*mi + p*mp], and a set of vectors (columns of B for Left, rows
// of B for Right).  Up to four vectors against more than one block take the chained
// solve (trsv_chain_kernel).  Large solves are halved while the product between the
// halves goes to the tensor cores (mod_gemm.cu).  The blocked, right-looking driver
// solves 64x64 diagonal blocks (trsm_diag_tile_kernel: 32 vectors per CTA, 8 rows per thread;
// trsm_diag_warp_kernel: a warp per vector for up to 2560 vectors) and applies
// each solved block to the rest of B with a GEMM.  The
// diagonal solve uses the column-sweep (axpy) form rather than the
// reference's dot form, and multiplies by the reciprocal of the diagonal
// instead of dividing; the result agrees to rounding.
#include "common.cuh"

#include <stdlib.h>

#include <atomic>

namespace fg {
namespace {

constexpr int TRSM_NB = 64;      // diagonal block size
constexpr int TRSM_VPC = 32;     // vectors per CTA
constexpr int TRSM_THREADS = 256;
constexpr int TRSM_RPT = TRSM_NB * TRSM_VPC / TRSM_THREADS;   // rows per thread (8)

// D[p][r] = M(r, p) of an nr x np block (zeros up to 64 x 64), 8 loads in flight
// per thread, along whichever index is contiguous.
template <int NT, typename T>
__device__ __forceinline__ void stage_block(T (*D)[TRSM_NB + 1], const T *__restrict__ M, long long mi, long long mp,
                                            int nr, int np) {
    const int t = threadIdx.x;
#pragma unroll 1
    for (int e0 = 0; e0 < TRSM_NB * TRSM_NB; e0 += 8 * NT) {
        T v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int e = e0 + j * NT + t, lo = e % TRSM_NB, hi = e / TRSM_NB;
            const int r = mi == 1 ? lo : hi, p = mi == 1 ? hi : lo;
            v[j] = r < nr && p < np ? M[r * mi + p * mp] : T(0);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int e = e0 + j * NT + t, lo = e % TRSM_NB, hi = e / TRSM_NB;
            if (mi == 1) D[hi][lo] = v[j];
            else D[lo][hi] = v[j];
        }
    }
}

// Row scaling of a staged FP64 diagonal block by the reciprocals of its diagonal:
// the substitution then has one FP64 instruction per step on its chain instead
// of two (a multiply by rinv_i after the sum).  M' = diag(rinv) M has each entry
// rounded once and b' = rinv b too, a componentwise backward error of the same
// form as with the multiply at the end; with the sums by blocks of the chained
// solve, the only user, the error of a solve (n = 100 to 1000, against extended
// precision) is 0.8 to 0.9 of the unscaled kernel's it replaced.  Only where no scaled entry leaves [2^-900, 2^900]
// (or is zero already): `scaled` is false otherwise and the block stays as it was.
// Only the solved triangle decides (LOWER: r > p): the other one may hold anything.
__device__ __forceinline__ int exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7FF; }
__device__ __forceinline__ bool mid_range(double x) {
    const int e = exp_field(x);
    return e >= 1023 - 900 && e <= 1023 + 900;
}
template <int NT, bool LOWER, typename T>
__device__ __forceinline__ bool scale_rows(T (*D)[TRSM_NB + 1], const T *rinv) {
    if (sizeof(T) != 8) return false;
    constexpr int PER = TRSM_NB * TRSM_NB / NT;
    T v[PER];
    bool ok = true;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = j * NT + threadIdx.x, r = e % TRSM_NB, p = e / TRSM_NB;
        v[j] = D[p][r] * rinv[r];
        ok &= mid_range((double)rinv[r]);
        if (LOWER ? r > p : r < p) ok &= mid_range((double)v[j]) || (__double_as_longlong((double)D[p][r]) << 1) == 0;
    }
    if (!__syncthreads_and(ok)) return false;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = j * NT + threadIdx.x;
        D[e / TRSM_NB][e % TRSM_NB] = v[j];
    }
    __syncthreads();
    return true;
}

// Substitution in the 32 x 32 diagonal sub-block at row o, one warp, lane = row
// (x: its entry).  A step is a shuffle of the finished entry and one FMA; an FP64
// warp instruction holds the scheduler's pipe for 64 clocks, so the chain is
// about 100 clocks a step.  MUL: times rinv[i] first (unscaled, not unit).
template <bool LOWER, bool MUL, typename T>
__device__ __forceinline__ void solve32(T &x, const T (*D)[TRSM_NB + 1], int o, const T *rinv) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int s = 0; s < 32; ++s) {
        const int i = LOWER ? s : 31 - s;
        T xi = __shfl_sync(0xffffffffu, x, i);
        if (MUL) {
            xi *= rinv[o + i];
            if (lane == i) x = xi;
        }
        if (LOWER ? lane > i : lane < i) x = fma(-D[o + i][o + lane], xi, x);
    }
}
template <bool LOWER, bool UNIT, typename T>
__device__ __forceinline__ void solve32_any(T &x, const T (*D)[TRSM_NB + 1], int o, const T *rinv, bool scaled) {
    if (UNIT || scaled) solve32<LOWER, false>(x, D, o, rinv);
    else solve32<LOWER, true>(x, D, o, rinv);
}

// Finite in all lanes (FP64: the exponents of two values, below 2^(limit + 1)).
template <typename T>
__device__ __forceinline__ bool all_below(T a, T b, int limit) {
    return __all_sync(0xffffffffu, exp_field((double)a) <= 1023 + limit && exp_field((double)b) <= 1023 + limit);
}

// One warp's vector by the plain substitution with the block as it is in memory: for
// a finite right-hand side that the scaled block takes beyond the range, in b' = rinv b
// (then at least 2^1001) or in a sum.  x0, x1: rows lane and lane + 32.
template <bool LOWER, typename T>
__device__ __noinline__ void solve_unscaled(T &x0, T &x1, const T *M, long long mi, long long mp, int kb,
                                            const T *rinv) {
    const int lane = threadIdx.x & 31;
    for (int s = 0; s < kb; ++s) {
        const int i = LOWER ? s : kb - 1 - s;
        const T xi = __shfl_sync(0xffffffffu, i < 32 ? x0 : x1, i & 31) * rinv[i];
        if (lane == (i & 31)) (i < 32 ? x0 : x1) = xi;
        if ((LOWER ? lane > i : lane < i) && lane < kb) x0 = fma(-M[lane * mi + i * mp], xi, x0);
        const int r = lane + 32;
        if ((LOWER ? r > i : r < i) && r < kb) x1 = fma(-M[r * mi + i * mp], xi, x1);
    }
}

// Solves the kb x kb (kb <= 64) diagonal block M for 32 vectors per CTA.
// Lane l of every warp holds vector l; warp w holds the 8 consecutive rows
// of row block blk(w) in registers.  Column by column, the warp owning row i
// finishes x_i (times the precomputed 1/M(i,i) unless the diagonal is unit)
// and publishes it through a double-buffered shared slot; after one barrier
// the warps with rows still open below (lower) or above (upper) i update
// them.  A warp whose rows are all finished skips the step as a whole, so
// the FP64 instructions issued are about 1.1x the triangle's FMAs (the pipe
// issues 2 FP64 lanes per clock per SM, so this is the kernel's bound); the
// blocks are paired {0,7}, {1,6}, {2,5}, {3,4} on the warps that share a
// scheduler so the schedulers get equal work.  The 64 x 32 tile of X is
// staged through shared memory so that global loads and stores are
// coalesced whichever of the row or vector index is contiguous.
//
// CYCLIC, while no SM has two of these CTAs: a column's chain (update of the next
// row, its reciprocal, shared memory, the barrier) is then what bounds it, and with
// consecutive rows its owner stands behind its own eight FMAs, 64 clocks each.  Here
// warp w holds the rows w + 8 j, so that all schedulers share each column, and the
// next entry is published after one FMA: 33 against 39 us up to 4864 vectors.
// Beyond, the pipe is the bound and consecutive rows, whose finished warps drop out,
// are ahead (8000 vectors: 51 against 53 us, 16000: 90 against 99).  The same
// operations per element in the same order.
template <typename T, bool LOWER, bool UNIT, bool CYCLIC>
__global__ void __launch_bounds__(TRSM_THREADS)
trsm_diag_tile_kernel(int nb, const T *__restrict__ M0, long long mi, long long mp,
                      T *__restrict__ X0, long long xs, long long vs, int nvec) {
    __shared__ T Ms[TRSM_NB][TRSM_NB + 1];     // Ms[i][r] = M(r, i)
    __shared__ T Xs[TRSM_NB][TRSM_VPC + 1];    // Xs[r][v]
    __shared__ T rinv[TRSM_NB];
    __shared__ T xb[2][TRSM_VPC];
    const int t = threadIdx.x;
    const long long v0 = (long long)blockIdx.x * TRSM_VPC;
    const int nv = (int)((nvec - v0) < TRSM_VPC ? (nvec - v0) : TRSM_VPC);
    stage_block<TRSM_THREADS>(Ms, M0, mi, mp, nb, nb);
    // X tile: lanes run along whichever index is contiguous in memory
    for (int e = t; e < TRSM_NB * TRSM_VPC; e += TRSM_THREADS) {
        int r, v;
        if (xs == 1) { r = e % TRSM_NB; v = e / TRSM_NB; }
        else { v = e % TRSM_VPC; r = e / TRSM_VPC; }
        Xs[r][v] = (r < nb && v < nv) ? X0[(v0 + v) * vs + r * xs] : T(0);
    }
    __syncthreads();
    if (!UNIT && t < nb) rinv[t] = T(1) / Ms[t][t];
    const int v = t & 31, w = t >> 5;
    const int r0 = CYCLIC ? w : 8 * (w < 4 ? w : 11 - w), rs = CYCLIC ? 8 : 1;        // the warp's rows: r0 + rs j
    T x[TRSM_RPT];
#pragma unroll
    for (int j = 0; j < TRSM_RPT; ++j) x[j] = Xs[r0 + rs * j][v];
    __syncthreads();
    if (CYCLIC) {
        // finishes x_i, held in xj, and publishes it for step s
        auto publish = [&](T &xj, int i, int s) {
            if (!UNIT) xj *= rinv[i];
            xb[s & 1][v] = xj;
        };
        {
            const int i = LOWER ? 0 : nb - 1;
            if (w == (i & 7)) {
                T xi = x[0];                              // selects, as below
#pragma unroll
                for (int j = 1; j < TRSM_RPT; ++j) xi = (j == i >> 3) ? x[j] : xi;
                publish(xi, i, 0);
#pragma unroll
                for (int j = 0; j < TRSM_RPT; ++j) x[j] = (j == i >> 3) ? xi : x[j];
            }
        }
        __syncthreads();
        int s = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const int j0 = LOWER ? b : 7 - b, j1 = LOWER ? b + 1 : 6 - b;      // row block of i, the next one
#pragma unroll 1
            for (int q = 0; q < 8; ++q) {
                const int c = LOWER ? q : 7 - q, i = 8 * j0 + c, in = LOWER ? i + 1 : i - 1;
                if (i >= nb) continue;
                const T xi = xb[s & 1][v];
                const T *m = &Ms[i][w];
                ++s;
                if (q < 7) {
                    if (LOWER ? w > c : w < c) x[j0] = fma(-m[8 * j0], xi, x[j0]);
                    if (w == (in & 7) && in < nb) publish(x[j0], in, s);
                }
                if (b < 7) {
                    x[j1 & 7] = fma(-m[8 * (j1 & 7)], xi, x[j1 & 7]);
                    if (q == 7 && w == (in & 7) && in < nb) publish(x[j1 & 7], in, s);
                }
#pragma unroll
                for (int h = 2; h < 8; ++h) {
                    const int j = LOWER ? b + h : 7 - b - h;
                    if (j >= 0 && j < 8) x[j] = fma(-m[8 * j], xi, x[j]);
                }
                __syncthreads();
            }
        }
    } else {
        for (int s = 0; s < nb; ++s) {
            const int i = LOWER ? s : nb - 1 - s;
            if ((i >> 3) == (r0 >> 3)) {                  // warp-uniform: owner of row i
                // selects, not x[i & 7]: an indexed access would move x to local memory
                const int k = i & 7;
                T xi = x[0];
#pragma unroll
                for (int j = 1; j < TRSM_RPT; ++j) xi = (j == k) ? x[j] : xi;
                if (!UNIT) xi *= rinv[i];
#pragma unroll
                for (int j = 0; j < TRSM_RPT; ++j) x[j] = (j == k) ? xi : x[j];
                xb[s & 1][v] = xi;
            }
            __syncthreads();
            if (LOWER ? (r0 + 7 > i) : (r0 < i)) {          // warp-uniform: rows still open
                const T xi = xb[s & 1][v];
#pragma unroll
                for (int j = 0; j < TRSM_RPT; ++j) {
                    const int r = r0 + j;
                    if (LOWER ? (r > i && r < nb) : (r < i)) x[j] = fma(-Ms[i][r], xi, x[j]);
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < TRSM_RPT; ++j) Xs[r0 + rs * j][v] = x[j];
    __syncthreads();
    for (int e = t; e < TRSM_NB * TRSM_VPC; e += TRSM_THREADS) {
        int r, vv;
        if (xs == 1) { r = e % TRSM_NB; vv = e / TRSM_NB; }
        else { vv = e % TRSM_VPC; r = e / TRSM_VPC; }
        if (r < nb && vv < nv) X0[(v0 + vv) * vs + r * xs] = Xs[r][vv];
    }
}

// FP32, many vectors: one thread per vector, the 64 entries in registers, the
// block's columns broadcast from shared memory 16 bytes at a time.  FP32 has no
// pipe to spare lanes for, so the 2016 FMAs of a vector, independent within a
// column, run without barriers: 24 us for 16384 vectors with the tile kernel
// above (a barrier per column).  Same operations per element in the same order.
constexpr int TRSM32_VPC = 64;
template <bool LOWER, bool UNIT>
__global__ void __launch_bounds__(TRSM32_VPC)
trsm32_thread_kernel(int nb, const float *__restrict__ M0, long long mi, long long mp,
                     float *__restrict__ X0, long long xs, long long vs, int nvec) {
    __shared__ __align__(16) float Ms[TRSM_NB][TRSM_NB];       // Ms[i][r] = M(r, i)
    __shared__ float Xs[TRSM_NB][TRSM32_VPC + 1];              // staging: M, then X
    __shared__ float rinv[TRSM_NB];
    const int t = threadIdx.x;
    const long long v0 = (long long)blockIdx.x * TRSM32_VPC;
    const int nv = (int)((nvec - v0) < TRSM32_VPC ? (nvec - v0) : TRSM32_VPC);
    stage_block<TRSM32_VPC>(Xs, M0, mi, mp, nb, nb);
    __syncthreads();
#pragma unroll 8
    for (int i = 0; i < TRSM_NB; ++i) Ms[i][t] = Xs[i][t];
    if (!UNIT) rinv[t] = t < nb ? 1.0f / Xs[t][t] : 1.0f;
    __syncthreads();
    float *X = X0 + v0 * vs;
#pragma unroll 1
    for (int e0 = 0; e0 < TRSM_NB; e0 += 8) {
        float w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = xs == 1 ? t : e0 + j, v = xs == 1 ? e0 + j : t;
            w[j] = r < nb && v < nv ? X[r * xs + v * vs] : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) Xs[xs == 1 ? t : e0 + j][xs == 1 ? e0 + j : t] = w[j];
    }
    __syncthreads();
    float x[TRSM_NB];
#pragma unroll
    for (int r = 0; r < TRSM_NB; ++r) x[r] = Xs[r][t];
#pragma unroll
    for (int s = 0; s < TRSM_NB; ++s) {
        const int i = LOWER ? s : TRSM_NB - 1 - s;
        if (!UNIT) x[i] *= rinv[i];
#pragma unroll
        for (int q = 0; q < TRSM_NB / 4; ++q) {
            if (LOWER ? 4 * q + 3 <= i : 4 * q >= i) continue;
            const float4 m = *(const float4 *)&Ms[i][4 * q];
            const float mm[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int r = 4 * q + h;
                if (LOWER ? r > i : r < i) x[r] = fmaf(-mm[h], x[i], x[r]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < TRSM_NB; ++r) Xs[r][t] = x[r];
    __syncthreads();
#pragma unroll 8
    for (int e = 0; e < TRSM_NB; ++e) {
        const int r = xs == 1 ? t : e, v = xs == 1 ? e : t;
        if (r < nb && v < nv) X[r * xs + v * vs] = Xs[r][v];
    }
}
static_assert(TRSM32_VPC == TRSM_NB, "thread t stages row t of X");

// Fewer vectors: one warp per vector, lane l holding rows l and l + 32.  The two
// 32 x 32 diagonal sub-blocks are substituted (solve32), the block between them
// is 32 independent FMAs.  Four warps per CTA, one per scheduler: with eight, two
// shared an FP64 pipe and the launch took 20 us instead of about 8.
constexpr int TRSM_WARP_VECS = 4;      // warps (vectors) per CTA

// The warp kernel is the lower-latency choice while the tile kernel would
// run at most one CTA per SM (each tile CTA is ~17 us of FP64 pipe time):
// up to FLENS_GB300_TRSM_WARP_MAX vectors, default 2560.
int trsm_warp_max() {
    static int v = [] {
        const char *e = getenv("FLENS_GB300_TRSM_WARP_MAX");
        const int x = e ? atoi(e) : 0;
        return x > 0 ? x : 2560;
    }();
    return v;
}

template <typename T, bool LOWER, bool UNIT>
__global__ void __launch_bounds__(32 * TRSM_WARP_VECS)
trsm_diag_warp_kernel(int nb, const T *__restrict__ M0, long long mi, long long mp,
                      T *__restrict__ X0, long long xs, long long vs, int nvec,
                      const int *__restrict__ skip) {
    __shared__ T Ms[TRSM_NB][TRSM_NB + 1];     // Ms[i][r] = M(r, i)
    __shared__ T rinv[TRSM_NB];
    const int stop = skip ? *skip : 0;         // (tested at the end: its latency is hidden)
    const int lane = threadIdx.x & 31;
    const long long v = (long long)blockIdx.x * TRSM_WARP_VECS + (threadIdx.x >> 5);
    T *x = X0 + v * vs;
    const int r0 = lane, r1 = lane + 32;
    T x0 = v < nvec && r0 < nb ? x[r0 * xs] : T(0);
    T x1 = v < nvec && r1 < nb ? x[r1 * xs] : T(0);
    stage_block<32 * TRSM_WARP_VECS>(Ms, M0, mi, mp, nb, nb);
    __syncthreads();
    if (!UNIT) {
        if (threadIdx.x < TRSM_NB) rinv[threadIdx.x] = threadIdx.x < nb ? T(1) / Ms[threadIdx.x][threadIdx.x] : T(1);
        __syncthreads();
    }
    if (v >= nvec) return;
    // (rows scaled by the reciprocals, as in the chained solve, would save a
    // multiply per step but raised the error of a 64-row solve by 4 to 15%)
    T &xa = LOWER ? x0 : x1, &xb = LOWER ? x1 : x0;        // solved first, second
    const int oa = LOWER ? 0 : 32, ob = 32 - oa;
    solve32<LOWER, !UNIT>(xa, Ms, oa, rinv);
#pragma unroll
    for (int s = 0; s < 32; ++s) {
        const int i = LOWER ? s : 31 - s;
        xb = fma(-Ms[oa + i][ob + lane], __shfl_sync(0xffffffffu, xa, i), xb);
    }
    solve32<LOWER, !UNIT>(xb, Ms, ob, rinv);
    if (stop) return;
    if (r0 < nb) x[r0 * xs] = x0;
    if (r1 < nb) x[r1 * xs] = x1;
}

// ------------------------------------------------------------------------
// Few vectors (<= 4) against a triangle of more than one block, in ONE launch:
// CTA s solves the s-th 64-row block in solve order (the first block for a
// lower triangle, the last for an upper one).  It applies the blocks solved
// before it as they are published -- staging each off-diagonal block of M
// before it waits, so the read overlaps the wait -- then solves its own
// diagonal block with one warp per vector and publishes it (release store of
// the call's epoch into its flag; acquire spins with an iteration limit).
// The launch is cooperative, so every CTA is resident and no wait can depend
// on a CTA that has not started.  This replaces the 2 x blocks launches of
// the blocked driver for the trs solves with one right-hand side.
constexpr int CH_NB = 64;
constexpr int CH_MAXV = 4;
constexpr int CH_THREADS = 256;

// spin limit of the next chained solve when it is made to stall (0: none)
std::atomic<unsigned> g_stall_next_chain{0};

__device__ __forceinline__ void ch_release(unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ch_acquire(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// spin_limit bounds every wait (kSpinLimit when 0).  stall != 0 is the
// failure-detection test: block 0 first waits for a flag value that nothing
// publishes, so it gives up, sets the status word and returns, and every
// block after it gives up in turn.
template <typename T, bool LOWER, bool UNIT>
__global__ void __launch_bounds__(CH_THREADS)
trsv_chain_kernel(int ka, const T *__restrict__ M0, long long mi, long long mp, T *X0, long long xs,
                  long long vs, int nvec, unsigned long long *flags, unsigned long long epoch,
                  int *status, unsigned spin_limit, int stall) {
    __shared__ T Mb[CH_NB][CH_NB + 1];                 // Mb[p][r] = M(R0 + r, K0 + p)
    __shared__ T Md[CH_NB][CH_NB + 1];                 // the diagonal block, same layout
    __shared__ T xk[CH_MAXV][CH_NB];
    __shared__ T part[CH_THREADS / CH_NB][CH_MAXV][CH_NB];
    __shared__ T rinv[CH_NB];
    __shared__ int s_abort;
    const int nblk = gridDim.x, s = blockIdx.x, tid = threadIdx.x;
    const int b = LOWER ? s : nblk - 1 - s;
    const int R0 = b * CH_NB, kb = min(CH_NB, ka - R0);
    const int r = tid & (CH_NB - 1), q = tid / CH_NB;    // row; 16-column quarter
    const unsigned limit = spin_limit ? spin_limit : kSpinLimit;
    if (tid == 0) {
        s_abort = 0;
        if (stall && s == 0) {
            // its own flag never holds epoch + 1 during this launch
            unsigned spins = 0;
            while (ch_acquire(&flags[0]) != epoch + 1) {
                if (++spins > limit) {
                    atomicOr(status, kDevBarrierTimeout);
                    s_abort = 1;
                    break;
                }
                if (spins > 32) __nanosleep(64);
            }
        }
    }
    T acc[CH_MAXV];
#pragma unroll
    for (int v = 0; v < CH_MAXV; ++v) acc[v] = T(0);

    auto stage = [&](T (*D)[CH_NB + 1], int K0, int kk) {
        stage_block<CH_THREADS>(D, M0 + R0 * mi + K0 * mp, mi, mp, kb, kk);
    };
    // the diagonal block, its reciprocals and the scaling of its rows do not
    // depend on other blocks: off the critical path, before any wait
    stage(Md, R0, kb);
    __syncthreads();
    if (s_abort) return;
    bool scaled = false;
    if (!UNIT) {
        if (tid < CH_NB) rinv[tid] = tid < kb ? T(1) / Md[tid][tid] : T(1);
        __syncthreads();
        scaled = scale_rows<CH_THREADS, LOWER>(Md, rinv);
    }

    for (int s2 = 0; s2 < s; ++s2) {
        const int k = LOWER ? s2 : nblk - 1 - s2;
        const int K0 = k * CH_NB, kk = min(CH_NB, ka - K0);
        stage(Mb, K0, kk);
        if (tid == 0) {
            unsigned spins = 0;
            while (ch_acquire(&flags[s2]) != epoch) {
                if (++spins > limit) {
                    atomicOr(status, kDevBarrierTimeout);
                    s_abort = 1;
                    break;
                }
                if (spins > 256) __nanosleep(32);
            }
        }
        __syncthreads();
        if (s_abort) return;
        // block k of x, final (L2 reads: an L1 line could predate the solve)
        for (int e = tid; e < nvec * CH_NB; e += CH_THREADS) {
            const int v = e / CH_NB, p = e % CH_NB;
            xk[v][p] = p < kk ? __ldcg(&X0[v * vs + (K0 + p) * xs]) : T(0);
        }
        __syncthreads();
        // each block's 16 products summed on their own, then added to the
        // running sum: (16 + blocks) roundings per row instead of 16 * blocks
        // (this matters for the FP32 solves of the refinement)
#pragma unroll
        for (int v = 0; v < CH_MAXV; ++v) {
            if (v < nvec) {
                T blk = T(0);
#pragma unroll 4
                for (int p = q * 16; p < q * 16 + 16; ++p) blk = fma(Mb[p][r], xk[v][p], blk);
                acc[v] += blk;
            }
        }
        __syncthreads();                                   // Mb and xk are restaged next
    }
#pragma unroll
    for (int v = 0; v < CH_MAXV; ++v) part[q][v][r] = acc[v];
    __syncthreads();
    // The block itself: warp v substitutes the first 32 rows of vector v (in solve
    // order), four warps form the 32 x 32 product with them, warp v substitutes
    // the other 32.  (One warp doing all 64 rows issued two to three FP64
    // instructions per step on one scheduler's pipe: 11.5 us a block, now about 6.)
    const int warp = tid >> 5, lane = tid & 31;
    const int oa = LOWER ? 0 : 32, ob = 32 - oa;
    T xa = T(0), xb = T(0), ba = T(0), bb = T(0);      // solution, right-hand side
    bool plain = false;
    if (warp < nvec) {
        const T *x = X0 + warp * vs + (long long)R0 * xs;
        auto rhs = [&](int rr) -> T {
            if (rr >= kb) return T(0);
            return x[rr * xs] - ((part[0][warp][rr] + part[1][warp][rr]) + (part[2][warp][rr] + part[3][warp][rr]));
        };
        xa = rhs(oa + lane);
        xb = rhs(ob + lane);
        ba = xa;
        bb = xb;
        if (scaled) {
            xa *= rinv[oa + lane];
            xb *= rinv[ob + lane];
            plain = !all_below(xa, xb, 1000) && all_below(ba, bb, 1023);
        }
        solve32_any<LOWER, UNIT>(xa, Md, oa, rinv, scaled);
        xk[warp][oa + lane] = xa;
    }
    __syncthreads();
    // (part is free: its first 32 rows take the product's four partial sums)
    for (int v = warp >> 2; v < nvec; v += CH_THREADS / 128) {
        const int g = warp & 3;
        T sum = T(0);
#pragma unroll
        for (int j = 0; j < 8; ++j) sum = fma(Md[oa + 8 * g + j][ob + lane], xk[v][oa + 8 * g + j], sum);
        part[g][v][lane] = sum;
    }
    __syncthreads();
    if (warp < nvec) {
        xb -= (part[0][warp][lane] + part[1][warp][lane]) + (part[2][warp][lane] + part[3][warp][lane]);
        solve32_any<LOWER, UNIT>(xb, Md, ob, rinv, scaled);
        T *x = X0 + warp * vs + (long long)R0 * xs;
        if (scaled && (plain || (!all_below(xa, xb, 1023) && all_below(ba, bb, 1023)))) {
            T &lo = LOWER ? ba : bb, &hi = LOWER ? bb : ba;
            solve_unscaled<LOWER>(lo, hi, M0 + R0 * (mi + mp), mi, mp, kb, rinv);
            xa = ba;
            xb = bb;
        }
        if (oa + lane < kb) x[(oa + lane) * xs] = xa;
        if (ob + lane < kb) x[(ob + lane) * xs] = xb;
    }
    __syncthreads();
    if (tid == 0) ch_release(&flags[s], epoch);
}

// Returns kErrUnsupported when the chained solve does not apply (too many
// blocks to keep resident, or more than the flag array holds).
template <typename T>
int launch_chain(int ka, const T *M0, long long mi, long long mp, bool lowerM, bool unit, T *X0,
                 long long xs, long long vs, int nvec, cudaStream_t stream,
                 const ChainFixed *fx) {
    const int nblk = ceil_div(ka, CH_NB);
    static int per_sm = -1;
    if (per_sm < 0) {
        int bps = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, trsv_chain_kernel<T, true, false>,
                                                          CH_THREADS, 0) != cudaSuccess) {
            cudaGetLastError();
            bps = 0;
        }
        per_sm = bps;
    }
    if ((long long)per_sm * num_sms() < nblk) return kErrUnsupported;
    unsigned long long *flags = nullptr, epoch = 0;
    int *status = nullptr;
    if (fx) {
        // caller-supplied flags: cleared in stream order, one fixed epoch
        if (nblk > fx->cap) return kErrUnsupported;
        FG_CUDA(cudaMemsetAsync(fx->flags, 0, sizeof(unsigned long long) * nblk, stream));
        flags = fx->flags;
        epoch = 1;
        status = fx->status;
    } else {
        int st = workspace_flags(stream, nblk, &flags, &epoch);
        if (st != kOk) return st;
        // a recorded launch publishes the same epoch at every replay: cleared before each
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) cudaGetLastError();
        if (cap != cudaStreamCaptureStatusNone)
            FG_CUDA(cudaMemsetAsync(flags, 0, sizeof(unsigned long long) * nblk, stream));
        Workspace *w = workspace_for(stream, 0);
        if (!w) return kErrAlloc;
        status = w->status;
    }
    // failure-detection test hook (flens_gb300_test_stall_next_chain)
    unsigned spin_limit = 0;
    int stall = 0;
    {
        const unsigned lim = g_stall_next_chain.exchange(0);
        if (lim) {
            spin_limit = lim;
            stall = 1;
        }
    }
    void *args[] = {&ka, &M0, &mi, &mp, &X0, &xs, &vs, &nvec, &flags, &epoch, &status,
                    &spin_limit, &stall};
    KTimer kt(kFamTrsv, stream, (double)ka * ka * nvec,
              (double)sizeof(T) * ka * (double)ka / 2.0 + 16.0 * ka * nvec);
    const void *fn;
    if (lowerM) fn = unit ? (const void *)trsv_chain_kernel<T, true, true>
                          : (const void *)trsv_chain_kernel<T, true, false>;
    else fn = unit ? (const void *)trsv_chain_kernel<T, false, true>
                   : (const void *)trsv_chain_kernel<T, false, false>;
    FG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(nblk), dim3(CH_THREADS), args, 0, stream));
    return kOk;
}

// Chained solves on (FLENS_GB300_TRSV_CHAIN=0 turns them off).
bool chain_enabled() {
    static bool on = [] {
        const char *e = getenv("FLENS_GB300_TRSV_CHAIN");
        return !(e && atoi(e) == 0);
    }();
    return on;
}

template <typename T>
int launch_diag(int kb, const T *M0, long long mi, long long mp, bool lowerM, bool unit,
                T *X0, long long xs, long long vs, int nvec, const int *skip, cudaStream_t stream) {
    KTimer kt(kFamTrsm, stream, (double)kb * kb * nvec, 16.0 * (double)kb * nvec);
    if (nvec <= trsm_warp_max() || skip) {     // (only this kernel looks at skip)
        const int grid = ceil_div(nvec, TRSM_WARP_VECS);
#define FG_WARP(L, U) trsm_diag_warp_kernel<T, L, U><<<grid, 32 * TRSM_WARP_VECS, 0, stream>>>(kb, M0, mi, mp, X0, xs, vs, nvec, skip)
        if (lowerM) { if (unit) FG_WARP(true, true); else FG_WARP(true, false); }
        else { if (unit) FG_WARP(false, true); else FG_WARP(false, false); }
#undef FG_WARP
    } else if constexpr (sizeof(T) == 4) {
        const int grid = ceil_div(nvec, TRSM32_VPC);
#define FG_THREAD(L, U) trsm32_thread_kernel<L, U><<<grid, TRSM32_VPC, 0, stream>>>(kb, M0, mi, mp, X0, xs, vs, nvec)
        if (lowerM) { if (unit) FG_THREAD(true, true); else FG_THREAD(true, false); }
        else { if (unit) FG_THREAD(false, true); else FG_THREAD(false, false); }
#undef FG_THREAD
    } else {
        const int grid = ceil_div(nvec, TRSM_VPC);
#define FG_TILE(L, U, C) trsm_diag_tile_kernel<T, L, U, C><<<grid, TRSM_THREADS, 0, stream>>>(kb, M0, mi, mp, X0, xs, vs, nvec)
#define FG_TILE_C(L, U) if (cyclic) FG_TILE(L, U, true); else FG_TILE(L, U, false)
        const bool cyclic = grid <= num_sms();
        if (lowerM) { if (unit) { FG_TILE_C(true, true); } else { FG_TILE_C(true, false); } }
        else { if (unit) { FG_TILE_C(false, true); } else { FG_TILE_C(false, false); } }
#undef FG_TILE_C
#undef FG_TILE
    }
    FG_CUDA(cudaGetLastError());
    return kOk;
}

template <typename T>
int gemm_t(char ta, char tb, int m, int n, int k, T alpha, const T *A, int ldA, const T *B,
           int ldB, T beta, T *C, int ldC, bool fixed, cudaStream_t s);
template <>
int gemm_t<double>(char ta, char tb, int m, int n, int k, double alpha, const double *A, int ldA,
                   const double *B, int ldB, double beta, double *C, int ldC, bool fixed,
                   cudaStream_t s) {
    // caller-supplied scratch (fixed): no product that allocates its own
    return (fixed ? dgemm_fp64_launch : dgemm_launch)(ta, tb, m, n, k, alpha, A, ldA, B, ldB, beta, C, ldC, s);
}
template <>
int gemm_t<float>(char ta, char tb, int m, int n, int k, float alpha, const float *A, int ldA,
                  const float *B, int ldB, float beta, float *C, int ldC, bool, cudaStream_t s) {
    return sgemm_launch(ta, tb, m, n, k, alpha, A, ldA, B, ldB, beta, C, ldC, s);
}

}  // namespace

template <typename T>
int trsm_launch_t(char side, char upLo, char transA, char diag, int m, int n,
                  T alpha, const T *A, int ldA, T *B, int ldB, cudaStream_t stream,
                  const ChainFixed *fx = nullptr, const int *skip = nullptr) {
    if (m == 0 || n == 0) return kOk;
    const bool left = (side == 'L' || side == 'l');
    const bool lowerA = (upLo == 'L' || upLo == 'l');
    const bool nT = (transA == 'N' || transA == 'n');
    const int unit = (diag == 'U' || diag == 'u') ? 1 : 0;
    const int ka = left ? m : n;
    const int nvec = left ? n : m;
    bool lowerM;
    long long mi, mp;
    if (left) {
        lowerM = lowerA ^ (!nT);
        mi = nT ? 1 : ldA;
        mp = nT ? ldA : 1;
    } else {
        lowerM = lowerA ^ nT;
        mi = nT ? ldA : 1;
        mp = nT ? 1 : ldA;
    }
    const long long xs = left ? 1 : ldB;
    const long long vs = left ? ldB : 1;
    trace("dtrsm %c%c%c%c m=%d n=%d (effective %s, %d vectors)", side, upLo, transA,
          diag, m, n, lowerM ? "lower" : "upper", nvec);

    const int nblk = ceil_div(ka, TRSM_NB);
    bool done = false;
    if (nvec <= CH_MAXV && nblk >= 2 && chain_enabled()) {
        const int st = launch_chain<T>(ka, A, mi, mp, lowerM, unit != 0, B, xs, vs, nvec, stream, fx);
        if (st == kOk) done = true;
        else if (st != kErrUnsupported) return st;
    }
    // Large FP64 solves by halves: T11 X1 = B1, B2 -= T21 X1, T22 X2 = B2.  The
    // products are as deep as the halves and go to the tensor cores
    // (mod_gemm.cu); 64-deep updates would read and write all of B for each.
    if (!done && sizeof(T) == 8 && !fx && nblk >= 4) {
        const int h = (nblk / 2) * TRSM_NB;            // first half in storage order
        if (mod_gemm_wins(left ? ka - h : m, left ? n : ka - h, h, 0)) {
            const T *A22 = A + h + (size_t)h * ldA;
            T *B2 = left ? B + h : B + (size_t)h * ldB;
            const int h2 = ka - h;
            auto solve = [&](bool second) -> int {
                return trsm_launch_t<T>(side, upLo, transA, diag, left ? (second ? h2 : h) : m,
                                        left ? n : (second ? h2 : h), T(1), second ? A22 : A, ldA, second ? B2 : B,
                                        ldB, stream);
            };
            // the stored off-diagonal block of the triangle; op() of it is
            // transposed exactly when op(A) is
            const T *Ao = lowerA ? A + h : A + (size_t)h * ldA;
            const char op = nT ? 'N' : 'T';
            // solved first: the first half for an effective lower triangle
            int st = solve(!lowerM);
            if (st != kOk) return st;
            if (left)
                st = lowerM ? gemm_t<T>(op, 'N', h2, n, h, T(-1), Ao, ldA, B, ldB, T(1), B2, ldB, false, stream)
                            : gemm_t<T>(op, 'N', h, n, h2, T(-1), Ao, ldA, B2, ldB, T(1), B, ldB, false, stream);
            else
                st = lowerM ? gemm_t<T>('N', op, m, h2, h, T(-1), B, ldB, Ao, ldA, T(1), B2, ldB, false, stream)
                            : gemm_t<T>('N', op, m, h, h2, T(-1), B2, ldB, Ao, ldA, T(1), B, ldB, false, stream);
            if (st == kOk) st = solve(lowerM);
            if (st != kOk) return st;
            done = true;
        }
    }
    for (int s = 0; !done && s < nblk; ++s) {
        const int bi = lowerM ? s : nblk - 1 - s;
        const int k0 = bi * TRSM_NB;
        const int kb = (ka - k0) < TRSM_NB ? (ka - k0) : TRSM_NB;
        int st0 = launch_diag<T>(kb, A + k0 * mi + k0 * mp, mi, mp, lowerM, unit != 0, B + k0 * xs, xs,
                              vs, nvec, skip, stream);
        if (st0 != kOk) return st0;
        // rows still to solve: below the block (lower) or above it (upper)
        const int r0 = lowerM ? k0 + kb : 0;
        const int rn = lowerM ? ka - (k0 + kb) : k0;
        if (rn <= 0) continue;
        int st;
        if (left) {
            // B[R,:] -= M[R,blk] * B[blk,:];  M(r,p) = A[r*mi + p*mp]
            const char opA = (mi == 1) ? 'N' : 'T';
            const T *Ap = (mi == 1) ? A + r0 + (size_t)k0 * ldA : A + k0 + (size_t)r0 * ldA;
            st = gemm_t<T>(opA, 'N', rn, n, kb, T(-1), Ap, ldA, B + k0, ldB, T(1), B + r0, ldB,
                           fx != nullptr, stream);
        } else {
            // B[:,R] -= B[:,blk] * M[R,blk]^T;  M[R,blk]^T(p,r) = A[r*mi + p*mp]
            const char opA = (mp == 1) ? 'N' : 'T';
            const T *Ap = (mp == 1) ? A + k0 + (size_t)r0 * ldA : A + r0 + (size_t)k0 * ldA;
            st = gemm_t<T>('N', opA, m, rn, kb, T(-1), B + (size_t)k0 * ldB, ldB, Ap, ldA, T(1),
                           B + (size_t)r0 * ldB, ldB, fx != nullptr, stream);
        }
        if (st != kOk) return st;
    }
    if (alpha != T(1)) {
        if (sizeof(T) == 8) return dscal_matrix_launch(m, n, (double)alpha, (double *)B, ldB, stream);
        return sscal_matrix_launch(m, n, (float)alpha, (float *)B, ldB, stream);
    }
    return kOk;
}

int dtrsm_launch(char side, char upLo, char transA, char diag, int m, int n, double alpha,
                 const double *A, int ldA, double *B, int ldB, cudaStream_t stream) {
    return trsm_launch_t<double>(side, upLo, transA, diag, m, n, alpha, A, ldA, B, ldB, stream);
}

int dtrsm_block_launch(char side, char upLo, char transA, char diag, int m, int n, double alpha,
                       const double *A, int ldA, double *B, int ldB, const int *skip, cudaStream_t stream) {
    if (((side == 'L' || side == 'l') ? m : n) > TRSM_NB || alpha != 1.0) return kErrUnsupported;
    return trsm_launch_t<double>(side, upLo, transA, diag, m, n, alpha, A, ldA, B, ldB, stream, nullptr, skip);
}

int dtrsm_launch_fixed(char side, char upLo, char transA, char diag, int m, int n, double alpha,
                       const double *A, int ldA, double *B, int ldB, const ChainFixed &fx,
                       cudaStream_t stream) {
    return trsm_launch_t<double>(side, upLo, transA, diag, m, n, alpha, A, ldA, B, ldB, stream, &fx);
}

int strsm_launch(char side, char upLo, char transA, char diag, int m, int n, float alpha,
                 const float *A, int ldA, float *B, int ldB, cudaStream_t stream) {
    return trsm_launch_t<float>(side, upLo, transA, diag, m, n, alpha, A, ldA, B, ldB, stream);
}

}  // namespace fg

// Failure-detection test hook: the next chained triangular solve (trs and
// trsm with at most 4 right-hand sides against more than one 64-row block)
// makes its first block wait for a flag that nothing sets, bounded by
// `spin_limit` spins, so that every block gives up and the stream's status
// word reports FLENS_GB300_ERR_TIMEOUT at the next flens_gb300_sync.  No
// fault, trap or unbounded wait is involved: the kernel returns and the
// context stays usable.
FG_API void flens_gb300_test_stall_next_chain(unsigned spin_limit) {
    fg::g_stall_next_chain.store(spin_limit);
}
