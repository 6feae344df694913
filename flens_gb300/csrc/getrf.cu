// getrf.cu -- blocked LU with partial pivoting (trf), its row interchanges
// (laswp) and solves (trs), FP64, column-major, 1-based pivots.
//
// Replaces, for double:
//   flens::lapack::trf  -> generic::trf_impl   flens/lapack/ge/trf.tcc:59-152
//   tf2 (panel)         -> generic::tf2_impl   flens/lapack/ge/tf2.tcc:56-136
//   laswp               -> generic::laswp_impl flens/lapack/la/laswp.tcc:54-93
//   trs                 -> generic::trs_impl   flens/lapack/ge/trs.tcc:59-109
//
// Orders (all asynchronous; the panel's width is the reference's ilaenv GETRF block
// size, flens/lapack/la/ilaenv.tcc:93-99):
//   - FP64 from 1024 columns on: outer blocks of 64 to 256 columns with look-ahead; a
//     block is factored by halves on a side stream while the previous block's update
//     runs (lookahead_nb).  FP32 storage from 2048 columns on: its outer blocks so.
//   - FP64, taller than 20,000 rows: the columns by halves, on one stream.
//   - smaller, and under stream capture: right-looking steps of 64 columns, the next
//     panel on the side stream beside the update.
// The pieces of each:
//     panel_cluster_kernel  panels of up to 6000 (FP32 13,300) rows: one cluster of 16
//                       CTAs, exchange by st.async (below).
//     panel_kernel      taller ones: cooperative grid, up to one CTA per SM; the (m-j) x jb
//                       panel lives in shared memory split by rows.  Per
//                       column each CTA finds its best candidate (warp-shuffle
//                       argmax, first maximum wins), publishes it with the
//                       candidate row in its own slot (release store of a
//                       sequence number) and reads every CTA's slot (acquire,
//                       bounded wait), so all CTAs agree on the pivot without
//                       a separate barrier; then every CTA swaps, scales and
//                       applies the rank-1 update to its own rows.  At the end
//                       it turns the jb interchanges into a list of
//                       (destination row, source row) moves.  FP32 storage
//                       uses panel32_kernel: FP32 arithmetic, and the key
//                       published in one word with its sequence number.
//     laswp_pairs_kernel applies those moves to every column outside the
//                       panel, one warp per column (loads, then stores).
//     dtrsm_launch      U12 = L11^-1 A12
//     dgemm_launch      A22 -= A21 * U12 (large ones by residues, mod_gemm.cu)
//
// Unlike the reference, the GPU path always uses the blocked algorithm (the
// reference switches to tf2 when nb >= min(m,n), trf.tcc:87-91); the pivots and
// factors are the same in exact arithmetic.
#include "common.cuh"

#include <float.h>
#include <limits.h>
#include <stdlib.h>

#include <algorithm>
#include <type_traits>
#include <mutex>

namespace fg {
namespace {

constexpr int PANEL_THREADS = 256;
constexpr int PANEL_NB = 64;           // max panel width
constexpr int PANEL_GMAX = 256;        // max CTAs in a panel grid
constexpr int PANEL_RMIN = 32;         // min rows per CTA
constexpr size_t PANEL_SMEM_MAX = 200 * 1024;

// One exchange slot per CTA and per step parity.  A CTA publishes its pivot
// candidate (|value|, row, the row's jb panel entries) and, if it owns panel
// row jj, that row; `seq` is written last with release semantics.
struct PanelSlot {
    unsigned long long seq;
    unsigned long long key;    // pivot key of the candidate (see pivot_key)
    int idx;
    int pad;
    double row[PANEL_NB];
    double rowjj[PANEL_NB];
};

struct PanelScratch {
    PanelSlot *slots;   // [2][GMAX]
    int *swap_cnt;      // [1]
    int *swap_dst;      // [2*NB]
    int *swap_src;      // [2*NB]
};

constexpr size_t kSlotBytes = 2 * (size_t)PANEL_GMAX * sizeof(PanelSlot);

size_t panel_scratch_bytes() { return kSlotBytes + 256 + 4 * PANEL_NB * sizeof(int) + 1024; }

PanelScratch carve_panel_scratch(void *base) {
    char *p = (char *)base;
    PanelScratch s;
    s.slots = (PanelSlot *)p;
    p += kSlotBytes;
    s.swap_cnt = (int *)p;
    p += 256;
    s.swap_dst = (int *)p;
    p += 2 * PANEL_NB * sizeof(int);
    s.swap_src = (int *)p;
    return s;
}

__device__ __forceinline__ void st_release(unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Pivot keys are integers, so the pivot search never touches the FP64 pipe
// (2 instructions per clock per SM on this part): |x| of a double orders
// like its bit pattern with the sign cleared.  0 = no candidate, 1 = NaN
// (loses to every number: iamax's `>` is false for NaN), |x| bits + 2
// otherwise.  (key, row) "better than": larger key; on equal keys the
// smaller row, which is cxxblas iamax's first-maximum rule
// (cxxblas/level1/iamax.tcc:52-56).
constexpr unsigned long long kKeyNone = 0ull;

__device__ __forceinline__ unsigned long long pivot_key(double x) {
    const unsigned long long a = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
    return a > 0x7ff0000000000000ull ? 1ull : a + 2ull;
}

// Named barrier 1 over `count` threads: the producer warp arrives without
// waiting, the consumers wait until every participant has arrived.
__device__ __forceinline__ void named_bar_arrive(int id, int count) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void named_bar_sync(int id, int count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

__device__ __forceinline__ bool better(unsigned long long k1, int i1, unsigned long long k2, int i2) {
    return k1 > k2 || (k1 == k2 && i1 < i2);
}

// Warp-wide argmax of (key, row) with three redux.sync: the largest high
// word, then the largest low word among those lanes, then the smallest row
// among the lanes holding that key.  Every lane gets the result; all 32
// lanes must call it.
__device__ __forceinline__ void warp_argmax(unsigned long long &k, int &i) {
    const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    const unsigned cand = (hi == mhi && lo == mlo) ? (unsigned)i : 0xffffffffu;
    i = (int)__reduce_min_sync(0xffffffffu, cand);
    k = ((unsigned long long)mhi << 32) | mlo;
}

// Block 0, warp 0 of a panel (all 32 lanes): the jb interchanges of the
// panel at column j0 (ipiv, written by this warp's lane 0 during the panel)
// as a list of (destination row, source row) moves, compacted to the moves
// that change something, into ps.swap_dst / swap_src / swap_cnt.
__device__ __forceinline__ void panel_moves(int jb, int j0, const int *ipiv, PanelScratch ps,
                                            int *s_list_row, int *s_list_src, int lane) {
    for (int i = lane; i < jb; i += 32) {
        s_list_row[i] = j0 + i;
        s_list_src[i] = j0 + i;
    }
    __syncwarp();
    int cnt = jb;
    for (int i = 0; i < jb; ++i) {
        const int p = ipiv[j0 + i] - 1;
        int pos;
        if (p < j0 + jb) {
            pos = p - j0;
        } else {
            int found = -1;
            for (int base = jb; base < cnt; base += 32) {
                const int e = base + lane;
                const unsigned hit = __ballot_sync(0xffffffffu, e < cnt && s_list_row[e] == p);
                if (hit) { found = base + __ffs(hit) - 1; break; }
            }
            if (found < 0) {
                found = cnt;
                if (lane == 0) { s_list_row[cnt] = p; s_list_src[cnt] = p; }
                ++cnt;
            }
            pos = found;
        }
        __syncwarp();
        if (lane == 0 && pos != i) {
            const int t = s_list_src[i];
            s_list_src[i] = s_list_src[pos];
            s_list_src[pos] = t;
        }
        __syncwarp();
    }
    if (lane == 0) {
        int k = 0;
        for (int e = 0; e < cnt; ++e) {
            if (s_list_row[e] != s_list_src[e]) {
                ps.swap_dst[k] = s_list_row[e];
                ps.swap_src[k] = s_list_src[e];
                ++k;
            }
        }
        *ps.swap_cnt = k;
    }
}

// Panel factorisation, tf2 semantics (flens/lapack/ge/tf2.tcc:56-136).
// A points at the panel's top-left element A(j,j); the panel is mp x jb.
// CTA b owns panel rows [b*R, min(mp,(b+1)*R)), kept in shared memory as
// S[c*R + r].  With at most 128 rows a CTA gives each row W = 2, 4 or 8
// lanes (interleaved columns); with more rows thread t owns local rows t,
// t+256, ... and updates them at once.  Block barriers per column: one to
// collect the warps' candidates, one after the cross-CTA poll, one to hand
// the pivot to every thread.  Warp 0 does the cross-CTA exchange.
// Two builds: DEFER (lanes per row and most of each column's rank-1 update
// deferred past the next column's candidate search, see [E2] below; about
// 120 registers per thread) for panels that run alone or beside a small
// update, and the immediate update within 64 registers for panels beside a
// large look-ahead GEMM (74 registers, 256 threads per CTA): at 102
// registers only one GEMM CTA fitted beside the panel instead of two (the
// n = 8192 LU: 325.9 against 322.8 ms per solve), and capping the deferred
// build instead slowed the split-update LU's panels by 11%.
template <typename T, bool DEFER>
__global__ void __launch_bounds__(PANEL_THREADS, DEFER ? 1 : 4)
panel_kernel(T *__restrict__ A, int lda, int mp, int jb, int j0,
             int *__restrict__ ipiv, int *__restrict__ info, int *__restrict__ status,
             PanelScratch ps, int R, unsigned long long epoch) {
    extern __shared__ double S[];
    constexpr int NW = PANEL_THREADS / 32;
    __shared__ double prow[PANEL_NB], orow[PANEL_NB];
    __shared__ unsigned long long red_k[NW], red_k2[NW];
    __shared__ int red_i[NW], red_i2[NW];
    __shared__ int s_gs, s_abort;
    __shared__ double s_pv, s_rinv;
    __shared__ int s_list_row[2 * PANEL_NB], s_list_src[2 * PANEL_NB];

    const int b = blockIdx.x, G = gridDim.x, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int rb = b * R;
    const int re = min(mp, rb + R);
    const int nr = max(0, re - rb);
    // lanes per row in the update: 8, 4 or 2 while nr * W fits the CTA
    const int W = nr <= 32 ? 8 : nr <= 64 ? 4 : nr <= 128 ? 2 : 1;

    for (int e = tid; e < nr * jb; e += PANEL_THREADS) {
        const int r = e % nr, c = e / nr;
        S[c * R + r] = A[(size_t)(rb + r) + (size_t)c * lda];
    }
    if (tid == 0) s_abort = 0;
    __syncthreads();

    // pivot keys of column 0 over the owned rows (later columns: computed
    // during the update)
    unsigned long long nbk = kKeyNone;
    int nbi = INT_MAX;
    for (int r = tid; r < nr; r += PANEL_THREADS) {
        const unsigned long long key = pivot_key(S[r]);
        if (better(key, rb + r, nbk, nbi)) { nbk = key; nbi = rb + r; }
    }

    // Deferred update (DEFER and W > 1): after the pivot of column jj is
    // known, each
    // row gets its swap, its multiplier l and the update of column jj + 1
    // (whose pivot keys the next search needs); the update of columns
    // >= jj + 2 waits until the next column's candidates are published, so
    // it runs while the other CTAs publish and this CTA polls.  Warp 0
    // publishes the candidate rows with those columns computed on the fly,
    // by the same FMA the deferred update stores: the factors are bitwise
    // those of the undeferred order.
    const bool lanes = W > 1, defer = DEFER && lanes;
    const double *dP = nullptr;          // pivot row of the pending update
    int d_jj = -1, d_gs = -1;            // its column and pivot row (-1: none)
    bool d_swap = false;
    bool pend = false, pend_gs = false;  // this thread's row has a pending update
    double pend_l = 0.0;
    for (int jj = 0; jj < jb; ++jj) {
        const int par = jj & 1;
        const unsigned long long want = epoch * 128ull + (unsigned long long)jj + 1ull;
        // -- [A] this CTA's candidate among its rows g >= jj
        unsigned long long k = nbk;
        int i = nbi;
        warp_argmax(k, i);
        if (lane == 0) { red_k[warp] = k; red_i[warp] = i; }
        __syncthreads();                                             // B1
        if (warp == 0) {
            // -- [B] publish the candidate row (and row jj if owned); the
            // release store by lane 0 after __syncwarp orders the warp's slot
            // writes before the sequence number
            k = lane < NW ? red_k[lane] : kKeyNone;
            i = lane < NW ? red_i[lane] : INT_MAX;
            warp_argmax(k, i);
            PanelSlot *mine = &ps.slots[par * PANEL_GMAX + b];
            // entry c of local row x, final (the pending update applied)
            auto fin = [&](int x, int c) -> double {
                if (d_jj < 0 || c < d_jj + 2) return S[c * R + x];
                const double src = (d_swap && rb + x == d_gs) ? orow[c] : S[c * R + x];
                return fma(-dP[c], S[d_jj * R + x], src);
            };
            // both rows into registers (jb <= 64: two entries per lane)
            // before the other warps may store their pending updates
            const bool has_i = i != INT_MAX, has_jj = jj >= rb && jj < re;
            double vi[2] = {0.0, 0.0}, vj[2] = {0.0, 0.0};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = lane + 32 * h;
                if (c < jb) {
                    if (has_i) vi[h] = fin(i - rb, c);
                    if (has_jj) vj[h] = fin(jj - rb, c);
                }
            }
            if (defer) named_bar_arrive(1, PANEL_THREADS);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = lane + 32 * h;
                if (c < jb) {
                    if (has_i) mine->row[c] = vi[h];
                    if (has_jj) mine->rowjj[c] = vj[h];
                }
            }
            if (lane == 0) {
                mine->key = k;
                mine->idx = i;
            }
            __syncwarp();
            if (lane == 0) st_release(&mine->seq, want);
        } else if (defer) {
            named_bar_sync(1, PANEL_THREADS);
        }
        // -- [E2] the pending update of column jj - 1: columns >= jj + 1
        if (pend) {
            const int r = tid / W, q = tid % W;
            const double *old = pend_gs ? orow : nullptr;
            int c = d_jj + 2 + q;
            for (; c + 3 * W < jb; c += 4 * W) {
                double v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = old ? old[c + u * W] : S[(c + u * W) * R + r];
#pragma unroll
                for (int u = 0; u < 4; ++u) S[(c + u * W) * R + r] = fma(-dP[c + u * W], pend_l, v[u]);
            }
            for (; c < jb; c += W) S[c * R + r] = fma(-dP[c], pend_l, old ? old[c] : S[c * R + r]);
            pend = false;
        }
        // -- [C] thread t < G waits for slot t of this step and reads it
        unsigned long long gk = kKeyNone;
        int gi = INT_MAX;
        if (tid < G) {
            const PanelSlot *sl = &ps.slots[par * PANEL_GMAX + tid];
            unsigned spins = 0;
            while (ld_acquire(&sl->seq) != want) {
                if (++spins > kSpinLimit) {
                    atomicOr(status, kDevBarrierTimeout);
                    s_abort = 1;
                    break;
                }
                if (spins > 32) __nanosleep(32);
            }
            gk = __ldcg(&sl->key);
            gi = __ldcg(&sl->idx);
        }
        if (warp * 32 < G) {                                          // warp-uniform
            warp_argmax(gk, gi);
            if (lane == 0) { red_k2[warp] = gk; red_i2[warp] = gi; }
        }
        __syncthreads();                                             // B2
        if (s_abort) return;
        if (warp == 0) {
            const int nw = (G + 31) / 32;
            gk = lane < nw ? red_k2[lane] : kKeyNone;
            gi = lane < nw ? red_i2[lane] : INT_MAX;
            warp_argmax(gk, gi);
            // -- [D] the old row jj and the winner's row, one round trip;
            // lane 0 settles the pivot (iamax starts from element jj: if it
            // is NaN nothing compares greater and jj is the pivot,
            // cxxblas/level1/iamax.tcc:50-57) and its reciprocal once
            const PanelSlot *sj = &ps.slots[par * PANEL_GMAX + jj / R];
            const PanelSlot *sw = &ps.slots[par * PANEL_GMAX + gi / R];
            for (int c = lane; c < jb; c += 32) {
                orow[c] = ld_cg(&sj->rowjj[c]);
                prow[c] = ld_cg(&sw->row[c]);
            }
            __syncwarp();
            if (lane == 0) {
                const double ajj = orow[jj];
                const int gs = isnan(ajj) ? jj : gi;
                const double pv = (gs == jj) ? ajj : prow[jj];
                s_gs = gs;
                s_pv = pv;
                s_rinv = (pv != 0.0 && fabs(pv) >= DBL_MIN) ? 1.0 / pv : 0.0;
                if (b == 0) {
                    ipiv[j0 + jj] = j0 + gs + 1;
                    if (pv == 0.0 && *info == 0) *info = j0 + jj + 1;
                }
            }
        }
        __syncthreads();                                             // B3
        const int gs = s_gs;
        const double pv = s_pv, rinv = s_rinv;
        const bool swap = (pv != 0.0) && (gs != jj);
        const double *P = (gs == jj) ? orow : prow;                  // new row jj

        // -- [E] per owned row: interchange, scaling, rank-1 update of the
        // columns > jj (deferred beyond jj + 1 when W > 1), and the pivot key
        // for column jj+1
        nbk = kKeyNone;
        nbi = INT_MAX;
        if (lanes) {
            // W lanes per row (nr * W <= 256: one row per lane group), lane q
            // of the group taking columns q, q + W, ...: the chain of
            // dependent shared-memory updates per thread is W times shorter.
            // The group's first lane reads the multiplier and broadcasts it
            // (all 32 lanes of every warp take part in the shuffle).
            const int r = tid / W, q = tid % W;
            const bool act = r < nr;
            const int g = rb + r;
            const bool to_jj = act && swap && g == jj, from_gs = act && swap && g == gs;
            double l0 = 0.0;
            if (act && q == 0) l0 = from_gs ? orow[jj] : S[jj * R + r];
            double l = __shfl_sync(0xffffffffu, l0, lane & ~(W - 1));
            if (to_jj) {
                for (int c = q; c < jb; c += W) S[c * R + r] = P[c];
            } else if (act && g > jj) {
                if (from_gs)
                    for (int c = q; c < jj; c += W) S[c * R + r] = orow[c];
                if (pv != 0.0) l = (rinv != 0.0) ? l * rinv : l / pv;
                if (q == 0 && pv != 0.0) S[jj * R + r] = l;
                const double *old = from_gs ? orow : nullptr;
                if (defer) {
                    // column jj + 1 and its key now, the rest in [E2]
                    if (q == 0 && jj + 1 < jb) {
                        const int c = jj + 1;
                        const double v = fma(-P[c], l, old ? old[c] : S[c * R + r]);
                        S[c * R + r] = v;
                        nbk = pivot_key(v);
                        nbi = g;
                    }
                    pend = jj + 2 + q < jb;
                    pend_gs = from_gs;
                    pend_l = l;
                } else {
                    int c = jj + 1 + q;
                    for (; c + 3 * W < jb; c += 4 * W) {
                        double v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) v[u] = old ? old[c + u * W] : S[(c + u * W) * R + r];
#pragma unroll
                        for (int u = 0; u < 4; ++u) S[(c + u * W) * R + r] = fma(-P[c + u * W], l, v[u]);
                    }
                    for (; c < jb; c += W) S[c * R + r] = fma(-P[c], l, old ? old[c] : S[c * R + r]);
                    if (q == 0 && jj + 1 < jb) {
                        nbk = pivot_key(S[(jj + 1) * R + r]);
                        nbi = g;
                    }
                }
            }
            if (defer) {
                dP = P;
                d_jj = jj;
                d_gs = gs;
                d_swap = swap;
            }
        } else
        for (int r = tid; r < nr; r += PANEL_THREADS) {
            const int g = rb + r;
            if (swap && g == jj) {
                for (int c = 0; c < jb; ++c) S[c * R + r] = P[c];
            } else if (swap && g == gs) {
                for (int c = 0; c < jb; ++c) S[c * R + r] = orow[c];
            }
            if (g > jj) {
                double l = S[jj * R + r];
                if (pv != 0.0) {
                    l = (rinv != 0.0) ? l * rinv : l / pv;
                    S[jj * R + r] = l;
                }
                for (int c = jj + 1; c < jb; ++c) S[c * R + r] = fma(-P[c], l, S[c * R + r]);
                if (jj + 1 < jb) {
                    const unsigned long long key = pivot_key(S[(jj + 1) * R + r]);
                    if (better(key, g, nbk, nbi)) { nbk = key; nbi = g; }
                }
            }
        }
    }
    __syncthreads();

    for (int e = tid; e < nr * jb; e += PANEL_THREADS) {
        const int r = e % nr, c = e / nr;
        A[(size_t)(rb + r) + (size_t)c * lda] = (T)S[c * R + r];
    }

    // -- block 0, warp 0: the jb interchanges as (dst, src) row moves.
    if (b == 0 && tid < 32) panel_moves(jb, j0, ipiv, ps, s_list_row, s_list_src, lane);
}

// ---- the panel of the FP32-storage LU ---------------------------------------
// Same algorithm and thread layout as panel_kernel, in FP32 arithmetic (the
// reference's tf2 instantiated for float: slamch's safe minimum is FLT_MIN)
// and with a shorter exchange.  A float's pivot key fits in 32 bits, so each
// CTA publishes its candidate as ONE 64-bit word, (sequence << 32) | key,
// stored as soon as the CTA's argmax is known and before anything else; the
// load that finds a slot current also returns its key, so the pivot is
// settled after one round trip through L2 instead of a release store that
// waits for the rows, a sequence poll and a dependent key load.  The rows
// (candidate and row jj) and the candidate's index follow under their own
// release-stored sequence word, and only the two rows the pivot needs are
// waited for.  Equal keys go to the lower CTA, whose rows come first: with
// each CTA's own first maximum this is iamax's first-maximum rule.
struct PanelSlot32 {
    unsigned long long head;   // (sequence << 32) | pivot key (pivot_key32)
    unsigned long long rseq;   // sequence, release-stored after row/rowjj/idx
    int idx;
    int pad[3];
    float row[PANEL_NB];
    float rowjj[PANEL_NB];
};
static_assert(2 * PANEL_GMAX * sizeof(PanelSlot32) <= kSlotBytes, "FP32 slots fit the exchange area");

// 0 = no candidate, 1 = NaN, |x| bits + 2 otherwise (at most 0x7f800002)
__device__ __forceinline__ unsigned long long pivot_key32(float x) {
    const unsigned a = __float_as_uint(x) & 0x7fffffffu;
    return a > 0x7f800000u ? 1ull : (unsigned long long)a + 2ull;
}

__device__ __forceinline__ void st_relaxed(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

template <bool DEFER>
__global__ void __launch_bounds__(PANEL_THREADS, DEFER ? 1 : 4)
panel32_kernel(float *__restrict__ A, int lda, int mp, int jb, int j0,
               int *__restrict__ ipiv, int *__restrict__ info, int *__restrict__ status,
               PanelScratch ps, int R, unsigned long long epoch) {
    extern __shared__ double S32_raw[];
    float *S = reinterpret_cast<float *>(S32_raw);
    constexpr int NW = PANEL_THREADS / 32;
    __shared__ float prow[PANEL_NB], orow[PANEL_NB];
    __shared__ unsigned long long red_k[NW], red_k2[NW];
    __shared__ int red_i[NW], red_i2[NW];
    __shared__ int s_gs, s_abort;
    __shared__ float s_pv, s_rinv;
    __shared__ int s_list_row[2 * PANEL_NB], s_list_src[2 * PANEL_NB];
    PanelSlot32 *slots = reinterpret_cast<PanelSlot32 *>(ps.slots);

    const int b = blockIdx.x, G = gridDim.x, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int rb = b * R;
    const int re = min(mp, rb + R);
    const int nr = max(0, re - rb);
    const int W = nr <= 32 ? 8 : nr <= 64 ? 4 : nr <= 128 ? 2 : 1;

    for (int e = tid; e < nr * jb; e += PANEL_THREADS) {
        const int r = e % nr, c = e / nr;
        S[c * R + r] = A[(size_t)(rb + r) + (size_t)c * lda];
    }
    if (tid == 0) s_abort = 0;
    __syncthreads();

    unsigned long long nbk = kKeyNone;
    int nbi = INT_MAX;
    for (int r = tid; r < nr; r += PANEL_THREADS) {
        const unsigned long long key = pivot_key32(S[r]);
        if (better(key, rb + r, nbk, nbi)) { nbk = key; nbi = rb + r; }
    }

    const bool lanes = W > 1, defer = DEFER && lanes;
    const float *dP = nullptr;
    int d_jj = -1, d_gs = -1;
    bool d_swap = false;
    bool pend = false, pend_gs = false;
    float pend_l = 0.0f;
    for (int jj = 0; jj < jb; ++jj) {
        const int par = jj & 1;
        const unsigned long long want = epoch * 128ull + (unsigned long long)jj + 1ull;
        const unsigned want32 = (unsigned)want;
        // -- [A] this CTA's candidate among its rows g >= jj
        unsigned long long k = nbk;
        int i = nbi;
        warp_argmax(k, i);
        if (lane == 0) { red_k[warp] = k; red_i[warp] = i; }
        __syncthreads();                                             // B1
        if (warp == 0) {
            // -- [B] the key first, in one word with its sequence number;
            // then the rows under their own sequence word
            k = lane < NW ? red_k[lane] : kKeyNone;
            i = lane < NW ? red_i[lane] : INT_MAX;
            warp_argmax(k, i);
            PanelSlot32 *mine = &slots[par * PANEL_GMAX + b];
            if (lane == 0) st_relaxed(&mine->head, ((unsigned long long)want32 << 32) | k);
            auto fin = [&](int x, int c) -> float {
                if (d_jj < 0 || c < d_jj + 2) return S[c * R + x];
                const float src = (d_swap && rb + x == d_gs) ? orow[c] : S[c * R + x];
                return fmaf(-dP[c], S[d_jj * R + x], src);
            };
            const bool has_i = i != INT_MAX, has_jj = jj >= rb && jj < re;
            float vi[2] = {0.0f, 0.0f}, vj[2] = {0.0f, 0.0f};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = lane + 32 * h;
                if (c < jb) {
                    if (has_i) vi[h] = fin(i - rb, c);
                    if (has_jj) vj[h] = fin(jj - rb, c);
                }
            }
            if (defer) named_bar_arrive(1, PANEL_THREADS);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = lane + 32 * h;
                if (c < jb) {
                    if (has_i) mine->row[c] = vi[h];
                    if (has_jj) mine->rowjj[c] = vj[h];
                }
            }
            if (lane == 0) mine->idx = i;
            __syncwarp();
            if (lane == 0) st_release(&mine->rseq, want);
        } else if (defer) {
            named_bar_sync(1, PANEL_THREADS);
        }
        // -- [E2] the pending update of column jj - 1: columns >= jj + 1
        if (pend) {
            const int r = tid / W, q = tid % W;
            const float *old = pend_gs ? orow : nullptr;
            int c = d_jj + 2 + q;
            for (; c + 3 * W < jb; c += 4 * W) {
                float v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = old ? old[c + u * W] : S[(c + u * W) * R + r];
#pragma unroll
                for (int u = 0; u < 4; ++u) S[(c + u * W) * R + r] = fmaf(-dP[c + u * W], pend_l, v[u]);
            }
            for (; c < jb; c += W) S[c * R + r] = fmaf(-dP[c], pend_l, old ? old[c] : S[c * R + r]);
            pend = false;
        }
        // -- [C] thread t < G waits for the key word of slot t; the winner is
        // the largest key, the lower CTA on equal keys
        unsigned long long gk = kKeyNone;
        int gc = INT_MAX;
        if (tid < G) {
            const PanelSlot32 *sl = &slots[par * PANEL_GMAX + tid];
            unsigned spins = 0;
            unsigned long long h;
            while (((h = ld_acquire(&sl->head)) >> 32) != (unsigned long long)want32) {
                if (++spins > kSpinLimit) {
                    atomicOr(status, kDevBarrierTimeout);
                    s_abort = 1;
                    break;
                }
                if (spins > 32) __nanosleep(32);
            }
            gk = h & 0xffffffffull;
            gc = tid;
        }
        if (warp * 32 < G) {                                          // warp-uniform
            warp_argmax(gk, gc);
            if (lane == 0) { red_k2[warp] = gk; red_i2[warp] = gc; }
        }
        __syncthreads();                                             // B2
        if (s_abort) return;
        if (warp == 0) {
            const int nw = (G + 31) / 32;
            gk = lane < nw ? red_k2[lane] : kKeyNone;
            gc = lane < nw ? red_i2[lane] : INT_MAX;
            warp_argmax(gk, gc);
            // -- [D] the winner's row and row jj, once their owners have
            // stored them (bounded waits, every lane)
            const PanelSlot32 *sj = &slots[par * PANEL_GMAX + jj / R];
            const PanelSlot32 *sw = &slots[par * PANEL_GMAX + gc];
            bool ok = true;
            {
                unsigned spins = 0;
                while (ld_acquire(&sw->rseq) != want || ld_acquire(&sj->rseq) != want) {
                    if (++spins > kSpinLimit) {
                        ok = false;
                        break;
                    }
                    if (spins > 32) __nanosleep(32);
                }
            }
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) {
                    atomicOr(status, kDevBarrierTimeout);
                    s_abort = 1;
                }
            } else {
                for (int c = lane; c < jb; c += 32) {
                    orow[c] = __ldcg(&sj->rowjj[c]);
                    prow[c] = __ldcg(&sw->row[c]);
                }
                const int gi = __ldcg(&sw->idx);
                __syncwarp();
                if (lane == 0) {
                    const float ajj = orow[jj];
                    const int gs = isnan(ajj) ? jj : gi;
                    const float pv = (gs == jj) ? ajj : prow[jj];
                    s_gs = gs;
                    s_pv = pv;
                    s_rinv = (pv != 0.0f && fabsf(pv) >= FLT_MIN) ? 1.0f / pv : 0.0f;
                    if (b == 0) {
                        ipiv[j0 + jj] = j0 + gs + 1;
                        if (pv == 0.0f && *info == 0) *info = j0 + jj + 1;
                    }
                }
            }
        }
        __syncthreads();                                             // B3
        if (s_abort) return;
        const int gs = s_gs;
        const float pv = s_pv, rinv = s_rinv;
        const bool swap = (pv != 0.0f) && (gs != jj);
        const float *P = (gs == jj) ? orow : prow;                   // new row jj

        // -- [E] per owned row: interchange, scaling, rank-1 update of the
        // columns > jj (deferred beyond jj + 1 when W > 1), and the pivot key
        // for column jj+1
        nbk = kKeyNone;
        nbi = INT_MAX;
        if (lanes) {
            const int r = tid / W, q = tid % W;
            const bool act = r < nr;
            const int g = rb + r;
            const bool to_jj = act && swap && g == jj, from_gs = act && swap && g == gs;
            float l0 = 0.0f;
            if (act && q == 0) l0 = from_gs ? orow[jj] : S[jj * R + r];
            float l = __shfl_sync(0xffffffffu, l0, lane & ~(W - 1));
            if (to_jj) {
                for (int c = q; c < jb; c += W) S[c * R + r] = P[c];
            } else if (act && g > jj) {
                if (from_gs)
                    for (int c = q; c < jj; c += W) S[c * R + r] = orow[c];
                if (pv != 0.0f) l = (rinv != 0.0f) ? l * rinv : l / pv;
                if (q == 0 && pv != 0.0f) S[jj * R + r] = l;
                const float *old = from_gs ? orow : nullptr;
                if (defer) {
                    if (q == 0 && jj + 1 < jb) {
                        const int c = jj + 1;
                        const float v = fmaf(-P[c], l, old ? old[c] : S[c * R + r]);
                        S[c * R + r] = v;
                        nbk = pivot_key32(v);
                        nbi = g;
                    }
                    pend = jj + 2 + q < jb;
                    pend_gs = from_gs;
                    pend_l = l;
                } else {
                    int c = jj + 1 + q;
                    for (; c + 3 * W < jb; c += 4 * W) {
                        float v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) v[u] = old ? old[c + u * W] : S[(c + u * W) * R + r];
#pragma unroll
                        for (int u = 0; u < 4; ++u) S[(c + u * W) * R + r] = fmaf(-P[c + u * W], l, v[u]);
                    }
                    for (; c < jb; c += W) S[c * R + r] = fmaf(-P[c], l, old ? old[c] : S[c * R + r]);
                    if (q == 0 && jj + 1 < jb) {
                        nbk = pivot_key32(S[(jj + 1) * R + r]);
                        nbi = g;
                    }
                }
            }
            if (defer) {
                dP = P;
                d_jj = jj;
                d_gs = gs;
                d_swap = swap;
            }
        } else
        for (int r = tid; r < nr; r += PANEL_THREADS) {
            const int g = rb + r;
            if (swap && g == jj) {
                for (int c = 0; c < jb; ++c) S[c * R + r] = P[c];
            } else if (swap && g == gs) {
                for (int c = 0; c < jb; ++c) S[c * R + r] = orow[c];
            }
            if (g > jj) {
                float l = S[jj * R + r];
                if (pv != 0.0f) {
                    l = (rinv != 0.0f) ? l * rinv : l / pv;
                    S[jj * R + r] = l;
                }
                for (int c = jj + 1; c < jb; ++c) S[c * R + r] = fmaf(-P[c], l, S[c * R + r]);
                if (jj + 1 < jb) {
                    const unsigned long long key = pivot_key32(S[(jj + 1) * R + r]);
                    if (better(key, g, nbk, nbi)) { nbk = key; nbi = g; }
                }
            }
        }
    }
    __syncthreads();

    for (int e = tid; e < nr * jb; e += PANEL_THREADS) {
        const int r = e % nr, c = e / nr;
        A[(size_t)(rb + r) + (size_t)c * lda] = S[c * R + r];
    }

    // -- block 0, warp 0: the jb interchanges as (dst, src) row moves.
    if (b == 0 && tid < 32) panel_moves(jb, j0, ipiv, ps, s_list_row, s_list_src, lane);
}

// Row moves of a run of interchanges, built by one warp in registers: entry e =
// lane + 32 h (h < 4) says that row mv_row ends up holding row mv_src; entries 0 ..
// nb-1 are the rows r0 .. r0+nb-1 (nb <= 64), others are added as they come.
// One step: interchange of row r0 + i and row p.
__device__ __forceinline__ void move_init(int (&mv_row)[4], int (&mv_src)[4], int lane, int r0, int nb) {
#pragma unroll
    for (int h = 0; h < 4; ++h) mv_row[h] = mv_src[h] = (lane + 32 * h < nb) ? r0 + lane + 32 * h : -1;
}
__device__ __forceinline__ void move_step(int (&mv_row)[4], int (&mv_src)[4], int &mv_cnt, int lane, int i, int p,
                                          int r0, int nb) {
    int pos = p - r0;
    if (pos < 0 || pos >= nb) {
        pos = -1;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const unsigned hit = __ballot_sync(0xffffffffu, mv_row[h] == p);
            if (hit) pos = 32 * h + __ffs(hit) - 1;
        }
        if (pos < 0) {
            pos = mv_cnt++;
#pragma unroll
            for (int h = 0; h < 4; ++h)
                if (lane + 32 * h == pos) mv_row[h] = mv_src[h] = p;
        }
    }
    int a = 0, c = 0;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const int x = __shfl_sync(0xffffffffu, mv_src[h], i & 31);
        const int y = __shfl_sync(0xffffffffu, mv_src[h], pos & 31);
        if ((i >> 5) == h) a = x;
        if ((pos >> 5) == h) c = y;
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        if (lane + 32 * h == i) mv_src[h] = c;
        if (lane + 32 * h == pos) mv_src[h] = a;
    }
}
// The moves that change something, compacted into dst / src; returns their number.
__device__ __forceinline__ int move_store(const int (&mv_row)[4], const int (&mv_src)[4], int mv_cnt, int lane,
                                          int *dst, int *src) {
    int base = 0;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const bool mv = lane + 32 * h < mv_cnt && mv_row[h] != mv_src[h];
        const unsigned m = __ballot_sync(0xffffffffu, mv);
        if (mv) {
            const int e = base + __popc(m & ((1u << lane) - 1u));
            dst[e] = mv_row[h];
            src[e] = mv_src[h];
        }
        base += __popc(m);
    }
    return base;
}

// ---- the panel of one thread-block cluster ----------------------------------
// The same factorisation for panels whose rows fit the shared memory of one
// cluster of 16 CTAs (16 SMs).  A column costs a search, an exchange of the
// candidates and an update; across the whole grid the exchange goes through L2
// (about 3 us a column with its polls and fences), inside a cluster it is one
// st.async into every CTA's shared memory, which counts its bytes on the
// receiver's mbarrier: no flags, fences or polls of memory.  Per column:
//   - every CTA's candidate (largest key, first row) by redux and one block
//     barrier; the pending update of the candidate row applied on the fly;
//   - three warps send the candidate row, row jj (its owner) and key and row number
//     to every CTA; in FP64 a fourth sends the candidate's reciprocal after them,
//     so that the division runs while the rows travel;
//   - the rest of the previous column's update, a warp per 32 rows and group of
//     4-column quads, while the exchange is under way; it reaches only to the end of
//     the sub-panel of 16 columns (FP32);
//   - every warp settles the pivot from the 16 headers; a thread per row scales
//     its entry, updates column jj+1 and takes its key for the next search.
// After the last column of a sub-panel all columns beyond it take its 16 updates at
// once, from registers (their U rows are solved column by column meanwhile): in
// shared memory every entry is then read and written 1/16 as often.  Per element the
// operations and their order stay those of the column-by-column update.
// The interchange of a row is applied where its entries are next read and
// written by one warp after the next candidate is out.  Three exchange buffers: a
// CTA can send column jj+3 only after all have sent jj+2, which they do after
// their last read of column jj's buffer.
// Bound: the chain search - exchange - settle (about 2200 clocks a column), from
// about m = 2000 on the 16 SMs' FP64 pipes (m * 32 FMAs a column at 32 per
// clock); in FP32 shared memory from about m = 6000 on.  Measured per column
// against the grid panel: FP64 2.0 against 3.8 us at n = 500, 2.4 against 4.0 at
// 2000, 3.0 against 4.1 at 4096 (whole LU); FP32 n = 16384, panels of the LU 42.7
// against 59.8 ms.
constexpr int CP_CS = 16;                       // CTAs of the cluster
constexpr int CP_T = 512;                       // threads per CTA
constexpr int CP_NW = CP_T / 32;
// Rows per thread at most.  (A second one in FP64, for panels of 8192 to 12,700
// rows, made every column 7% slower at n = 500.)
template <typename T>
constexpr int CP_RPT = sizeof(T) == 8 ? 1 : 2;
constexpr int CP_NARROW = 32;                   // columns held for a panel of at most as many
// Columns of a sub-panel.  FP64 has none: its bound is the FP64 pipe, not shared
// memory, and the U rows, 15 dependent FP64 FMAs, made a column 12% slower.
template <typename T>
constexpr int CP_SB = sizeof(T) == 8 ? PANEL_NB : 16;

template <typename T>
struct ClusterBuf {                             // one exchange buffer
    T row[CP_CS][PANEL_NB];                     // candidate rows
    T rowjj[PANEL_NB];
    ulonglong2 head[CP_CS];                     // key, row
    double rinv[CP_CS];                         // FP64: 1 / candidate (0: divide)
};

template <typename T>
constexpr uint32_t cluster_bytes() {            // received per column
    return CP_CS * (PANEL_NB * sizeof(T) + 16 + (sizeof(T) == 8 ? 8 : 0)) + PANEL_NB * sizeof(T);
}

// Rows a cluster holds beside its static buffers, `cols` (64 or 32) columns wide (at
// most CP_RPT per thread).
template <typename T>
constexpr size_t cluster_rows_max(int cols) {
    const size_t bytes = 227 * 1024 - 2048 - 3 * sizeof(ClusterBuf<T>) - (CP_SB<T> % PANEL_NB) * PANEL_NB * sizeof(T);
    const size_t rows = bytes / (cols * sizeof(T));
    return (rows < CP_RPT<T> * CP_T ? rows : CP_RPT<T> * CP_T) * CP_CS;
}

__device__ __forceinline__ uint32_t cp_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cp_map(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cp_send16(uint32_t dst, uint32_t bar, unsigned long long a, unsigned long long b) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "l"(a), "l"(b), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cp_send8(uint32_t dst, uint32_t bar, unsigned long long a) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst), "l"(a),
                 "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cp_send_pair(uint32_t dst, uint32_t bar, double a, double b) {
    cp_send16(dst, bar, (unsigned long long)__double_as_longlong(a), (unsigned long long)__double_as_longlong(b));
}
__device__ __forceinline__ void cp_send_pair(uint32_t dst, uint32_t bar, float a, float b) {
    cp_send8(dst, bar, (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32));
}
__device__ __forceinline__ unsigned long long cp_key(double x) { return pivot_key(x); }
__device__ __forceinline__ unsigned long long cp_key(float x) { return pivot_key32(x); }
__device__ __forceinline__ double cp_rinv(double p) { return (p != 0.0 && fabs(p) >= DBL_MIN) ? 1.0 / p : 0.0; }
__device__ __forceinline__ float cp_rinv(float p) { return (p != 0.0f && fabsf(p) >= FLT_MIN) ? 1.0f / p : 0.0f; }
__device__ __forceinline__ double cp_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float cp_fma(float a, float b, float c) { return fmaf(a, b, c); }

// The lane holding the warp's largest key, the first on equal keys.
__device__ __forceinline__ int cp_best(unsigned long long k, double) {
    const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    return __ffs(__ballot_sync(0xffffffffu, hi == mhi && lo == mlo)) - 1;
}
__device__ __forceinline__ int cp_best(unsigned long long k, float) {      // keys below 2^32
    const unsigned lo = (unsigned)k, m = __reduce_max_sync(0xffffffffu, lo);
    return __ffs(__ballot_sync(0xffffffffu, lo == m)) - 1;
}

// Bounded wait of the whole block's threads on one phase of an mbarrier.
__device__ __forceinline__ bool cp_wait(uint32_t bar, uint32_t parity) {
    for (unsigned i = 0; i < (1u << 20); ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

template <typename T>
__global__ void __launch_bounds__(CP_T, 1)
panel_cluster_kernel(T *__restrict__ A, int lda, int mp, int jb, int j0, int *__restrict__ ipiv,
                     int *__restrict__ info, int *__restrict__ status, PanelScratch ps, int R) {
    extern __shared__ double S_raw[];
    T *S = reinterpret_cast<T *>(S_raw);
    __shared__ __align__(16) ClusterBuf<T> buf[3];
    constexpr int SB = CP_SB<T>;
    __shared__ __align__(16) T Us[SB < PANEL_NB ? SB : 1][PANEL_NB];   // U rows of the sub-panel, columns beyond it
    __shared__ unsigned long long bars[3];
    __shared__ unsigned long long red_k[2][CP_NW];
    __shared__ int red_i[2][CP_NW];
    __shared__ int s_abort;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x;                    // one cluster: the block index is the rank
    const int rb = b * R, nr = max(0, min(mp, rb + R) - rb);

    if (tid == 0) {
        for (int i = 0; i < 3; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cp_smem(&bars[i])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    // columns jb .. ncol - 1 take part in the updates: keep them defined
    const int ncol = jb <= CP_NARROW ? CP_NARROW : PANEL_NB;
    {
        const int nrb = (nr + 31) / 32;
        for (int u = warp; u < nrb * 4; u += CP_NW) {
            const int r = (u % nrb) * 32 + lane, c0 = u / nrb;
            if (r < nr)
#pragma unroll
                for (int h = 0; h < 16; ++h) {
                    const int c = c0 + 4 * h;
                    if (c < ncol) S[c * R + r] = c < jb ? A[(size_t)(rb + r) + (size_t)c * lda] : T(0);
                }
        }
    }
    __syncthreads();
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");

    // pivot keys of column 0: thread per row (rows tid, tid + 512)
    unsigned long long nbk = kKeyNone;
    int nbi = INT_MAX;
    for (int r = tid; r < nr; r += CP_T) {
        const unsigned long long key = cp_key(S[r]);
        if (better(key, rb + r, nbk, nbi)) { nbk = key; nbi = rb + r; }
    }

    // row moves of the interchanges, kept by CTA 0's last warp: entry e =
    // lane + 32 h is (row, source); the first jb rows are the panel's top
    int mv_row[4], mv_src[4], mv_cnt = jb;
    move_init(mv_row, mv_src, lane, j0, jb);

    // the column whose update is pending (-1: none), its pivot row and buffers
    // (d_end: end of the columns it covers, 0 after a bulk update; d_done: the
    // columns d_jj .. d_done of row d_gs hold newer values than dO)
    int d_jj = -1, d_gs = -1, d_end = 0, d_done = 0;
    bool d_swap = false;
    const T *dP = nullptr, *dO = nullptr;
    // deferred writes of the interchange of column d_jj: row d_jj <- dP, row
    // d_gs <- dO (its columns d_jj + 2 .. d_end - 1: by the pending update)
    auto write_swap = [&]() {
        if (!d_swap) return;
        const int rj = d_jj - rb, rg = d_gs - rb;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = lane + 32 * h;
            if (c < jb) {
                if (rj >= 0 && rj < nr && (c <= d_jj || d_end)) S[c * R + rj] = dP[c];
                if (rg >= 0 && rg < nr && (c < d_jj || (d_end && c >= d_end))) S[c * R + rg] = dO[c];
            }
        }
    };

    // U row jj of the sub-panel at s0 beyond it, from the pivot row P as exchanged (whose
    // entries there are not updated yet): warp half `w` takes 32 of the columns
    auto u_row = [&](int jj, int s0, int w, const T *P) {
        if constexpr (SB < PANEL_NB) {
        const int c = s0 + SB + 32 * w + lane;
        if (c >= PANEL_NB) return;
        T v = P[c];
        for (int t = s0; t < jj; ++t) v = cp_fma(-Us[t - s0][c], P[t], v);
        Us[jj - s0][c] = v;
        }
    };

    int bi = 0;                                  // buffer of this column
    uint32_t phase = 0;                          // its parity
    // rows are in the order of lanes, warps and CTAs: on equal keys the first lane
    // (warp, CTA) wins.  Not with two rows per thread.
    const bool ordered = nr <= CP_T;
    for (int jj = 0; jj < jb; ++jj) {
        const int s0 = jj & ~(SB - 1), s1 = s0 + SB;
        const bool bulk = SB < PANEL_NB && jj == s1 - 1 && s1 < jb;           // last column of a sub-panel
        // -- this CTA's candidate among its rows g >= jj
        unsigned long long k = nbk;
        int i = nbi;
        if (ordered) {
            const int w = cp_best(k, T(0));
            if (lane == w) { red_k[jj & 1][warp] = k; red_i[jj & 1][warp] = i; }
        } else {
            warp_argmax(k, i);
            if (lane == 0) { red_k[jj & 1][warp] = k; red_i[jj & 1][warp] = i; }
        }
        const uint32_t bar = cp_smem(&bars[bi]);
        if (tid == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                         "r"(cluster_bytes<T>())
                         : "memory");
        if (__syncthreads_or(s_abort)) break;                        // B1
        ClusterBuf<T> &cur = buf[bi];
        // Warps 0 and 1 send the candidate row and row jj, each lane two columns of
        // it to all CTAs; warp 2 the key and row number, a lane per CTA; warp 3 (FP64)
        // the reciprocal.  The others wait only until the rows are read.
        constexpr int NSEND = sizeof(T) == 8 ? 4 : 3;
        bool sent = false;
        if (warp < NSEND) {
            k = lane < CP_NW ? red_k[jj & 1][lane] : kKeyNone;
            i = lane < CP_NW ? red_i[jj & 1][lane] : INT_MAX;
            if (ordered) {
                const int w = cp_best(k, T(0));
                k = __shfl_sync(0xffffffffu, k, w);
                i = __shfl_sync(0xffffffffu, i, w);
            } else {
                warp_argmax(k, i);
            }
            // entry c of local row x with the pending interchange and update
            auto fin = [&](int x, int c) -> T {
                const bool sw = d_swap && rb + x == d_gs && (c < d_jj || c > d_done);
                const T v = sw ? dO[c] : S[c * R + x];
                return (c >= d_jj + 2 && c < d_end) ? cp_fma(-dP[c], S[d_jj * R + x], v) : v;
            };
            const bool has = warp == 0 ? i != INT_MAX : (jj >= rb && jj < rb + nr);
            if (warp < 2) {
                const int x = (warp == 0 ? i : jj) - rb;
                T v0 = T(0), v1 = T(0);
                if (has && 2 * lane < ncol) {
                    v0 = fin(x, 2 * lane);
                    v1 = fin(x, 2 * lane + 1);
                }
                __syncwarp();
                named_bar_arrive(1, CP_T);
                sent = true;
                if (warp == 0 || has) {
                    const uint32_t dst = cp_smem(warp == 0 ? &cur.row[b][2 * lane] : &cur.rowjj[2 * lane]);
#pragma unroll
                    for (int t = 0; t < CP_CS; ++t) cp_send_pair(cp_map(dst, t), cp_map(bar, t), v0, v1);
                }
                named_bar_sync(2, 64);           // both rows are read
            } else if (warp == 2) {
                if (lane < CP_CS)
                    cp_send16(cp_map(cp_smem(&cur.head[b]), lane), cp_map(bar, lane), k, (unsigned long long)(unsigned)i);
            } else {
                // (column jj is final; 0 where the CTA has no row left)
                const T pc = i != INT_MAX ? S[jj * R + i - rb] : T(0);
                named_bar_sync(1, CP_T);
                sent = true;
                const double r = (double)cp_rinv(pc);
                if (lane < CP_CS)
                    cp_send8(cp_map(cp_smem(&cur.rinv[b]), lane), cp_map(bar, lane),
                             (unsigned long long)__double_as_longlong(r));
            }
        }
        if (!sent) named_bar_sync(1, CP_T);
        // -- the pending update of column d_jj: columns d_jj + 2 .. d_end - 1
        if (d_end) {
            const int nrb = (nr + 31) / 32;
            const int ncg = nrb >= CP_NW ? 1 : CP_NW / max(nrb, 1);
            const int q0 = (d_jj + 2) >> 2, q1 = min(d_end, ncol) >> 2;
            for (int u = warp; u < nrb * ncg; u += CP_NW) {
                const int cg = u / nrb, r = (u - cg * nrb) * 32 + lane, g = rb + r;
                if (r < nr && g > d_jj) {
                    const T l = S[d_jj * R + r];
                    const bool sw = d_swap && g == d_gs;
                    // two quads at a time: eight loads before the first store
                    for (int q = q0 + cg; q < q1; q += 2 * ncg) {
                        const int qb = q + ncg < q1 ? q + ncg : q;
                        T p[8], v[8];
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            p[h] = dP[4 * q + h];
                            p[4 + h] = dP[4 * qb + h];
                        }
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            v[h] = sw ? dO[4 * q + h] : S[(4 * q + h) * R + r];
                            v[4 + h] = sw ? dO[4 * qb + h] : S[(4 * qb + h) * R + r];
                        }
#pragma unroll
                        for (int h = 0; h < 4; ++h)
                            if (4 * q + h >= d_jj + 2) S[(4 * q + h) * R + r] = cp_fma(-p[h], l, v[h]);
                        if (qb != q)
#pragma unroll
                            for (int h = 0; h < 4; ++h) S[(4 * qb + h) * R + r] = cp_fma(-p[4 + h], l, v[4 + h]);
                    }
                }
            }
            if (SB < PANEL_NB && s1 < jb && (warp == CP_NW - 4 || warp == CP_NW - 3)) u_row(d_jj, s0, warp - (CP_NW - 4), dP);
        }
        if (warp == CP_NW - 2) write_swap();
        // -- this thread's entries of columns jj and jj + 1 (its own writes)
        T c0[CP_RPT<T>], c1[CP_RPT<T>];
#pragma unroll
        for (int h = 0; h < CP_RPT<T>; ++h) {
            const int r = tid + h * CP_T;
            c0[h] = r < nr ? S[jj * R + r] : T(0);
            c1[h] = r < nr && jj + 1 < jb ? S[(jj + 1) * R + r] : T(0);
        }
        // -- the 16 candidates
        const bool arrived = cp_wait(bar, phase);
        if (!arrived) {
            atomicOr(status, kDevBarrierTimeout);
            s_abort = 1;
        }
        const ulonglong2 head = cur.head[lane & (CP_CS - 1)];
        const T ajj = cur.rowjj[jj];
        int src = cp_best(head.x, T(0)) & (CP_CS - 1);
        const int gi = (int)(unsigned)__shfl_sync(0xffffffffu, (unsigned)head.y, src);
        const bool jnan = cp_key(ajj) == 1ull;    // integer tests: no FP64 compares
        const bool own = jnan || gi < 0 || gi >= mp;              // (out of range: a wait gave up)
        const int gs = own ? jj : gi;
        const T *P = own ? cur.rowjj : cur.row[src], *O = cur.rowjj;
        const T pv = P[jj];
        const T rinv = jnan ? T(0) : sizeof(T) == 8 ? (T)cur.rinv[src] : cp_rinv(pv);
        const bool pnz = cp_key(pv) != 2ull, rnz = cp_key(rinv) != 2ull;
        const bool swap = pnz && gs != jj;
        // -- thread per row: scale, column jj + 1, next key
        nbk = kKeyNone;
        nbi = INT_MAX;
#pragma unroll
        for (int h = 0; h < CP_RPT<T>; ++h) {
            const int r = tid + h * CP_T, g = rb + r;
            if (r >= nr || g <= jj) continue;
            const bool sw = swap && g == gs;
            T l = sw ? O[jj] : c0[h];
            if (pnz) l = rnz ? l * rinv : l / pv;
            S[jj * R + r] = l;
            if (jj + 1 < jb && !bulk) {
                const T v = cp_fma(-P[jj + 1], l, sw ? O[jj + 1] : c1[h]);
                S[(jj + 1) * R + r] = v;
                const unsigned long long key = cp_key(v);
                if (better(key, g, nbk, nbi)) { nbk = key; nbi = g; }
            }
        }
        if constexpr (SB < PANEL_NB) if (bulk) {
            // -- the columns beyond the sub-panel, all its updates at once
            if (warp == CP_NW - 4 || warp == CP_NW - 3) u_row(jj, s0, warp - (CP_NW - 4), P);
            __syncthreads();
            const int nrb = (nr + 31) / 32;
            const int ncg = nrb >= CP_NW ? 1 : CP_NW / max(nrb, 1);
            const int q1 = (jb + 3) >> 2;
            for (int u = warp; u < nrb * ncg; u += CP_NW) {
                const int cg = u / nrb, r = (u - cg * nrb) * 32 + lane, g = rb + r;
                if (r >= nr || g < s0) continue;
                const bool sw = swap && g == gs;
                T l[SB];
#pragma unroll
                for (int t = 0; t < SB; ++t)
                    l[t] = g < s1 ? T(0) : (sw && t < SB - 1) ? O[s0 + t] : S[(s0 + t) * R + r];
                for (int q = (s1 >> 2) + cg; q < q1; q += ncg) {
                    T v[4];
                    if (g < s1) {                        // a pivot row: final
#pragma unroll
                        for (int h = 0; h < 4; ++h) v[h] = Us[g - s0][4 * q + h];
                    } else {
#pragma unroll
                        for (int h = 0; h < 4; ++h) v[h] = sw ? O[4 * q + h] : S[(4 * q + h) * R + r];
#pragma unroll
                        for (int t = 0; t < SB; ++t) {
                            T p[4];
#pragma unroll
                            for (int h = 0; h < 4; ++h) p[h] = Us[t][4 * q + h];
#pragma unroll
                            for (int h = 0; h < 4; ++h) v[h] = cp_fma(-p[h], l[t], v[h]);
                        }
                        if (q == (s1 >> 2)) {            // column s1, by the thread of this row
                            const unsigned long long key = cp_key(v[0]);
                            if (better(key, g, nbk, nbi)) { nbk = key; nbi = g; }
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 4; ++h) S[(4 * q + h) * R + r] = v[h];
                }
            }
        }
        d_jj = jj;
        d_gs = gs;
        d_swap = swap;
        d_end = bulk ? 0 : s1;
        d_done = bulk ? PANEL_NB : jj + 1;
        dP = P;
        dO = O;
        if (b == 0 && warp == CP_NW - 1) {
            if (lane == 0) {
                ipiv[j0 + jj] = j0 + gs + 1;
                if (!pnz && *info == 0) *info = j0 + jj + 1;
            }
            // the interchange jj <-> gs in the list of moves
            move_step(mv_row, mv_src, mv_cnt, lane, jj, j0 + gs, j0, jb);
        }
        if (++bi == 3) {
            bi = 0;
            phase ^= 1u;
        }
    }
    // the last interchange
    if (warp == CP_NW - 2 && d_jj >= 0) write_swap();
    __syncthreads();
    // no CTA leaves while others may still send to it
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    if (s_abort) return;
    {
        const int nrb = (nr + 31) / 32;
        for (int u = warp; u < nrb * 4; u += CP_NW) {
            const int r = (u % nrb) * 32 + lane, c0 = u / nrb;
            if (r < nr)
#pragma unroll
                for (int h = 0; h < 16; ++h) {
                    const int c = c0 + 4 * h;
                    if (c < jb) A[(size_t)(rb + r) + (size_t)c * lda] = S[c * R + r];
                }
        }
    }
    if (b == 0 && warp == CP_NW - 1) {
        const int base = move_store(mv_row, mv_src, mv_cnt, lane, ps.swap_dst, ps.swap_src);
        if (lane == 0) *ps.swap_cnt = base;
    }
}


// Apply the panel's row moves to columns [0, cSplit) and [cSplit+skip, ...),
// ncols columns in total; one warp per column.
template <typename T>
__global__ void __launch_bounds__(256)
laswp_pairs_kernel(T *__restrict__ A, int lda, int ncols, int cSplit, int skip,
                   const int *__restrict__ cntp, const int *__restrict__ dst,
                   const int *__restrict__ src) {
    __shared__ int s_dst[2 * PANEL_NB], s_src[2 * PANEL_NB];
    const int cnt = *cntp;
    if (cnt == 0) return;
    for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
        s_dst[e] = dst[e];
        s_src[e] = src[e];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= ncols) return;
    const int c = q < cSplit ? q : q + skip;
    T *col = A + (size_t)c * lda;
    T v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int e = lane + 32 * t;
        if (e < cnt) v[t] = col[s_src[e]];
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int e = lane + 32 * t;
        if (e < cnt) col[s_dst[e]] = v[t];
    }
}

// ---- laswp with an arbitrary pivot range (used by trs) ----------------------
// perm[r] = source row of row r after the interchanges i <-> piv(i) for
// i = k1..k2 (inc > 0) or k2..k1 (inc < 0).  The interchanges do not commute, but
// a run of 64 of them moves at most 128 rows: every warp builds the moves of one
// run in registers, 32 runs at a time, and four warps apply them to the
// permutation run by run (in shared memory when it fits).  One thread walking
// the pivots took 212 us at n = 4096; this takes about 20.
constexpr int LASWP_WARPS = 32, LASWP_RUN = 64;
constexpr int LASWP_SMEM = 176 * 1024;
__global__ void __launch_bounds__(32 * LASWP_WARPS)
laswp_perm_kernel(int nrows, int k1, int k2, const int *__restrict__ ipiv,
                  int inc, int *__restrict__ perm_g, int use_smem) {
    extern __shared__ int perm_s[];
    __shared__ int s_dst[LASWP_WARPS][2 * LASWP_RUN], s_src[LASWP_WARPS][2 * LASWP_RUN], s_cnt[LASWP_WARPS];
    int *perm = use_smem ? perm_s : perm_g;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int r = tid; r < nrows; r += blockDim.x) perm[r] = r;
    const int runs = (k2 - k1 + LASWP_RUN) / LASWP_RUN;
    for (int b0 = 0; b0 < runs; b0 += LASWP_WARPS) {
        const int run = b0 + warp;                     // in order of application
        if (run < runs) {
            const int c = inc > 0 ? run : runs - 1 - run;
            const int r0 = k1 - 1 + c * LASWP_RUN, nb = min(LASWP_RUN, k2 - r0);
            int pv[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) pv[h] = lane + 32 * h < nb ? ipiv[r0 + lane + 32 * h] - 1 : -1;
            int mv_row[4], mv_src[4], mv_cnt = nb;
            move_init(mv_row, mv_src, lane, r0, nb);
            for (int t = 0; t < nb; ++t) {
                const int i = inc > 0 ? t : nb - 1 - t;
                const int p = __shfl_sync(0xffffffffu, i < 32 ? pv[0] : pv[1], i & 31);
                if (p != r0 + i && p >= 0 && p < nrows) move_step(mv_row, mv_src, mv_cnt, lane, i, p, r0, nb);
            }
            const int cnt = move_store(mv_row, mv_src, mv_cnt, lane, s_dst[warp], s_src[warp]);
            if (lane == 0) s_cnt[warp] = cnt;
        }
        __syncthreads();
        if (warp < 4) {
            const int nr = min(LASWP_WARPS, runs - b0);
            for (int j = 0; j < nr; ++j) {
                const bool on = tid < s_cnt[j];
                const int v = on ? perm[s_src[j][tid]] : 0;
                named_bar_sync(1, 128);
                if (on) perm[s_dst[j][tid]] = v;
                named_bar_sync(1, 128);
            }
        }
        __syncthreads();
    }
    if (use_smem)
        for (int r = tid; r < nrows; r += blockDim.x) perm_g[r] = perm[r];
}

// tmp[:, c] = A[perm, c] for the first nrows rows
template <typename T>
__global__ void gather_rows_kernel(int nrows, int ncols, const T *__restrict__ A, int lda,
                                   const int *__restrict__ perm, T *__restrict__ tmp) {
    const size_t total = (size_t)nrows * ncols;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
         e += (size_t)gridDim.x * blockDim.x) {
        const size_t c = e / nrows, r = e % nrows;
        tmp[e] = A[(size_t)perm[r] + c * lda];
    }
}

template <typename T>
__global__ void copy_back_kernel(int nrows, int ncols, const T *__restrict__ tmp,
                                 T *__restrict__ A, int lda) {
    const size_t total = (size_t)nrows * ncols;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
         e += (size_t)gridDim.x * blockDim.x) {
        const size_t c = e / nrows, r = e % nrows;
        A[r + c * lda] = tmp[e];
    }
}

template <typename T>
int trsm_t(char side, char uplo, char ta, char diag, int m, int n, T alpha, const T *A, int ldA,
           T *B, int ldB, cudaStream_t s);
template <>
int trsm_t<double>(char side, char uplo, char ta, char diag, int m, int n, double alpha,
                   const double *A, int ldA, double *B, int ldB, cudaStream_t s) {
    return dtrsm_launch(side, uplo, ta, diag, m, n, alpha, A, ldA, B, ldB, s);
}
template <>
int trsm_t<float>(char side, char uplo, char ta, char diag, int m, int n, float alpha,
                  const float *A, int ldA, float *B, int ldB, cudaStream_t s) {
    return strsm_launch(side, uplo, ta, diag, m, n, alpha, A, ldA, B, ldB, s);
}
template <typename T>
int gemm_tt(char ta, char tb, int m, int n, int k, T alpha, const T *A, int ldA, const T *B,
            int ldB, T beta, T *C, int ldC, cudaStream_t s);
template <>
int gemm_tt<double>(char ta, char tb, int m, int n, int k, double alpha, const double *A, int ldA,
                    const double *B, int ldB, double beta, double *C, int ldC, cudaStream_t s) {
    return dgemm_launch(ta, tb, m, n, k, alpha, A, ldA, B, ldB, beta, C, ldC, s);
}
template <>
int gemm_tt<float>(char ta, char tb, int m, int n, int k, float alpha, const float *A, int ldA,
                   const float *B, int ldB, float beta, float *C, int ldC, cudaStream_t s) {
    return sgemm_launch(ta, tb, m, n, k, alpha, A, ldA, B, ldB, beta, C, ldC, s);
}

// The outer trailing update A22 -= L21 * U12 of the two-level LU: through the
// split GEMM for FP64 storage, on the tensor cores in `tc_kind` for FP32.
template <typename T>
int outer_update(int m, int n, int k, const T *L21, int ldL, const T *U12, int ldU, T *A22,
                 int ldA22, size_t ws0_off, int tc_kind, void *tc_buf, cudaStream_t s);
template <>
int outer_update<double>(int m, int n, int k, const double *L21, int ldL, const double *U12,
                         int ldU, double *A22, int ldA22, size_t ws0_off, int, void *,
                         cudaStream_t s) {
    return dgemm_split_launch_at('N', 'N', m, n, k, -1.0, L21, ldL, U12, ldU, 1.0, A22, ldA22, 0,
                                 nullptr, ws0_off, s);
}
template <>
int outer_update<float>(int m, int n, int k, const float *L21, int ldL, const float *U12, int ldU,
                        float *A22, int ldA22, size_t, int tc_kind, void *tc_buf, cudaStream_t s) {
    if (tc_kind < 0) {
        set_last_error("getrf: an FP32 outer update needs a tensor-core kind");
        return kErrUnsupported;
    }
    return tc_trailing_update(tc_kind, m, n, k, L21, ldL, U12, ldU, A22, ldA22, tc_buf, s);
}

// The FP32 panel (panel32_kernel) for FP32 storage: on unless
// FLENS_GB300_PANEL32=0, which factors FP32 panels with panel_kernel<float>
// (FP64 arithmetic on the FP32 values).
bool panel32_enabled() {
    static bool on = [] {
        const char *e = getenv("FLENS_GB300_PANEL32");
        return !(e && atoi(e) == 0);
    }();
    return on;
}

// Look-ahead in the blocked LU: on unless FLENS_GB300_LOOKAHEAD=0.
bool lookahead_enabled() {
    static bool on = [] {
        const char *e = getenv("FLENS_GB300_LOOKAHEAD");
        return !(e && atoi(e) == 0);
    }();
    return on;
}

// Width of the cluster panel at mp rows, 0: the grid panel.  64 as far as a
// cluster holds 64 columns (FP32: 13,300 rows; per column 1.7 us at 4096 rows, 3.0
// at 13,000, the grid panel 3.5), in FP64 up to 6000 rows, where its 16 SMs' FP64
// pipes come level with the grid panel's 4.1 us.  Beyond, 32 columns up to twice
// the rows where the panel runs beside an update (`beside`): the grid panel needs
// all SMs.  (Alone, 32-wide panels were no faster: half the pipe time per column,
// twice the launches.)  FLENS_GB300_PANEL_CLUSTER bounds the rows (0: never).
template <typename T>
int cluster_width(int mp, bool beside) {
    static int cap = [] {
        const char *e = getenv("FLENS_GB300_PANEL_CLUSTER");
        return e && *e ? atoi(e) : INT_MAX;
    }();
    const int wide = sizeof(T) == 8 ? 6000 : (int)cluster_rows_max<T>(PANEL_NB);
    if (mp > cap) return 0;
    if (mp <= wide) return PANEL_NB;
    return beside && mp <= (int)cluster_rows_max<T>(CP_NARROW) ? CP_NARROW : 0;
}

cudaLaunchConfig_t cluster_config(cudaLaunchAttribute *attr, size_t smem, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CP_CS);
    cfg.blockDim = dim3(CP_T);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = CP_CS;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Whether a cluster of 16 full-size CTAs can be resident on the device
// (16 SMs of one GPC); asked once per device.
template <typename T>
bool cluster_fits() {
    static int known[64];                         // 0: not asked, 1: yes, 2: no
    const int d = device_id();
    if (d < 0 || d >= 64) return false;
    int v = __atomic_load_n(&known[d], __ATOMIC_ACQUIRE);
    if (v == 0) {
        const size_t smem = std::max(cluster_rows_max<T>(PANEL_NB) / CP_CS * PANEL_NB,
                                     cluster_rows_max<T>(CP_NARROW) / CP_CS * CP_NARROW) * sizeof(T);
        const void *fn = (const void *)panel_cluster_kernel<T>;
        cudaLaunchAttribute attr;
        cudaLaunchConfig_t cfg = cluster_config(&attr, smem, nullptr);
        int n = 0;
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        v = n >= 1 ? 1 : 2;
        __atomic_store_n(&known[d], v, __ATOMIC_RELEASE);
        trace("getrf<%d>: clusters of %d CTAs resident: %d", (int)sizeof(T), CP_CS, n);
    }
    return v == 1;
}

// CTAs of a panel grid: at most one per SM and PANEL_GMAX, or
// FLENS_GB300_PANEL_CTAS when set (1..that bound).
int panel_ctas(int sms) {
    int cap = sms < PANEL_GMAX ? sms : PANEL_GMAX;
    static int env = [] {
        const char *e = getenv("FLENS_GB300_PANEL_CTAS");
        return e ? atoi(e) : 0;
    }();
    if (env >= 1 && env < cap) cap = env;
    return cap;
}

// Rows per CTA of a grid panel of mp rows, and its width: the reference's 64,
// narrowed only if a CTA's rows would not fit in shared memory (very tall
// matrices, few CTAs); 0 when no column does.
int grid_panel_rows(int mp, int gcap) {
    const int R = ceil_div(mp, gcap);
    return R < PANEL_RMIN ? PANEL_RMIN : R;
}
int grid_panel_width(int mp, int gcap, size_t elem_bytes) {
    const size_t R = (size_t)grid_panel_rows(mp, gcap);
    int nb = PANEL_NB;
    while (nb > 0 && R * nb * elem_bytes > PANEL_SMEM_MAX) nb >>= 1;
    return nb;
}

// SMs left to the side stream's cluster panel.
constexpr int kClusterSms = CP_CS;

// Outer block of the FP64 order with look-ahead (FLENS_GB300_LOOKAHEAD_NB, a
// multiple of 64).  A narrow block gets the next panel started sooner, a wide one
// makes the updates deeper.  Factorisations in ms with 64, 128 and 256 columns:
//   n    2000   3000   4000   4300   4600   5000   5500   6000   6500   7000   8192
//    64  5.92   10.1   16.0   18.4   20.9   24.9   30.3   36.7   44.4   53.2   78.1
//   128  6.47   11.1   16.6   18.5   20.4   23.5   27.2   31.1   35.9   41.2   56.0
//   256  6.95   11.8   17.3   19.2   21.1   23.7   27.4   30.6   34.6   39.1   50.8
// (halved without look-ahead: 7.7 at 2048, 28.5 at 5000, 60.0 at 8192).
int lookahead_nb(int mn) {
    static int nb = [] {
        const char *e = getenv("FLENS_GB300_LOOKAHEAD_NB");
        const int v = e ? atoi(e) : 0;
        return (v >= 64 && v <= 1024 && v % 64 == 0) ? v : 0;
    }();
    return nb > 0 ? nb : mn < 4400 ? 64 : mn < 5700 ? 128 : 256;
}

// Whether the FP64 LU takes outer blocks with look-ahead, or halves the columns
// (matrices too tall for cluster panels): its products then go to the tensor
// cores.  From 1024 columns on (n = 1000: 2.59 ms both ways).  Not for a stream
// under capture, whose products run on the FP64 pipe: there the right-looking
// order of 64-column steps is faster (n = 8192: 320 against 355 ms).
bool recursive_lu(int m, int n, cudaStream_t stream) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const int h = (m < n ? m : n) / 2;
    if (h < 512) return false;
    return cap == cudaStreamCaptureStatusNone && mod_gemm_wins(m - h, n - h, h, 0);
}

// Whether the FP32 LU with tensor-core updates takes its outer blocks with
// look-ahead.
bool sgetrf_lookahead(int m, int n, cudaStream_t stream) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return cap == cudaStreamCaptureStatusNone && (m < n ? m : n) >= 2048;
}

// Outer block of the split-update LU: FLENS_GB300_SPLIT_NB (a multiple of 64),
// else 512.
int split_outer_nb() {
    static int nb = [] {
        const char *e = getenv("FLENS_GB300_SPLIT_NB");
        const int v = e ? atoi(e) : 0;
        return (v >= 64 && v % 64 == 0) ? v : 512;
    }();
    return nb;
}

// Outer block of the tensor-core LU (FLENS_GB300_TC_NB, a multiple of 64; 64
// = one level): its trailing updates have this depth, so they read and write
// the FP32 C once per outer block instead of once per 64 columns.  At
// n = 16384 the updates took 49.8, 28.0 and 17.3 ms for 64, 128 and 256.
int tc_outer_nb() {
    static int nb = [] {
        const char *e = getenv("FLENS_GB300_TC_NB");
        const int v = e ? atoi(e) : 0;
        return (v >= 64 && v % 64 == 0) ? v : 256;
    }();
    return nb;
}

}  // namespace

template <typename T>
int laswp_launch_t(int nrows, int ncols, T *A, int ldA, int k1, int k2, const int *ipiv, int inc,
                   cudaStream_t stream) {
    if (nrows <= 0 || ncols <= 0 || k2 < k1) return kOk;
    const size_t permBytes = ((size_t)nrows * sizeof(int) + 255) / 256 * 256;
    const size_t tmpBytes = (size_t)nrows * ncols * sizeof(T);
    Workspace *w = workspace_for(stream, permBytes + tmpBytes);
    if (!w) return kErrAlloc;
    int *perm = (int *)w->buf;
    T *tmp = (T *)((char *)w->buf + permBytes);
    const int use_smem = (size_t)nrows * sizeof(int) <= LASWP_SMEM ? 1 : 0;
    if (use_smem) {
        static DeviceOnce once;
        const int st0 = set_smem_once(once, (const void *)laswp_perm_kernel, LASWP_SMEM);
        if (st0 != kOk) return st0;
    }
    KTimer kt(kFamLaswp, stream, 0.0, 4.0 * sizeof(T) * (double)nrows * ncols);
    laswp_perm_kernel<<<1, 1024, use_smem ? (size_t)nrows * sizeof(int) : 0, stream>>>(
        nrows, k1, k2, ipiv, inc, perm, use_smem);
    FG_CUDA(cudaGetLastError());
    const size_t total = (size_t)nrows * ncols;
    int blocks = (int)ceil_div(total, (size_t)256);
    if (blocks > num_sms() * 16) blocks = num_sms() * 16;
    gather_rows_kernel<T><<<blocks, 256, 0, stream>>>(nrows, ncols, A, ldA, perm, tmp);
    FG_CUDA(cudaGetLastError());
    copy_back_kernel<T><<<blocks, 256, 0, stream>>>(nrows, ncols, tmp, A, ldA);
    FG_CUDA(cudaGetLastError());
    return kOk;
}

// perm[r] = source row of row r after the interchanges ipiv(1..nrows): the
// forward laswp as one gather (used by the solves of the precision form).
int laswp_perm_launch(int nrows, const int *ipiv, int *perm, cudaStream_t stream) {
    if (nrows <= 0) return kOk;
    const int use_smem = (size_t)nrows * sizeof(int) <= LASWP_SMEM ? 1 : 0;
    if (use_smem) {
        static DeviceOnce once;
        const int st0 = set_smem_once(once, (const void *)laswp_perm_kernel, LASWP_SMEM);
        if (st0 != kOk) return st0;
    }
    KTimer kt(kFamLaswp, stream, 0.0, 8.0 * nrows);
    laswp_perm_kernel<<<1, 1024, use_smem ? (size_t)nrows * sizeof(int) : 0, stream>>>(
        nrows, 1, nrows, ipiv, 1, perm, use_smem);
    FG_CUDA(cudaGetLastError());
    return kOk;
}

int dlaswp_launch(int nrows, int ncols, double *A, int ldA, int k1, int k2, const int *ipiv,
                  int inc, cudaStream_t stream) {
    return laswp_launch_t<double>(nrows, ncols, A, ldA, k1, k2, ipiv, inc, stream);
}

int slaswp_launch(int nrows, int ncols, float *A, int ldA, int k1, int k2, const int *ipiv,
                  int inc, cudaStream_t stream) {
    return laswp_launch_t<float>(nrows, ncols, A, ldA, k1, k2, ipiv, inc, stream);
}

// Bytes of slot-0 workspace the blocked LU needs: the panel exchange area
// plus, for a tensor-core trailing update, its operand buffers.
size_t getrf_workspace_bytes(int m, int n, int tc_kind, int depth) {
    size_t b = (panel_scratch_bytes() + 255) / 256 * 256;
    if (tc_kind >= 0) b += tc_update_workspace_bytes(tc_kind, m, n, depth > PANEL_NB ? depth : PANEL_NB);
    return b;
}

// Blocked right-looking LU over storage T.  Panel, interchanges and the U12
// solve always run here; the trailing update A22 -= A21*U12 runs in T on the
// CUDA cores (tc_kind < 0) or, for T = float, on the tensor cores in the
// precision `tc_kind` (see tc_gemm.cu).
//
// split_nb > 0: two-level blocking.  The 64-column steps of an outer block
// of split_nb columns update only the columns of that block (their
// interchanges still reach every column); when the block is done,
// U12 = L11^-1 A12 for all columns to its right (trsm in T) and
// A22 -= L21 U12 with depth split_nb, through the split GEMM for T = double
// and on the tensor cores in `tc_kind` for T = float.  This is the order of
// LAPACK's dgetrf with a recursive panel; in exact arithmetic the factors
// and pivots are those of the right-looking loop.
//
// recursive: the columns are halved down to panels (left half, U12 by trsm,
// one product, right half), so that the products are as deep as they are
// wide and run on the tensor cores by residues (mod_gemm.cu), where a 64-deep
// update would only move C.
template <typename T>
int getrf_t(int m, int n, T *A, int ldA, int *ipiv, int *info, int tc_kind, int split_nb,
            cudaStream_t stream, bool recursive = false) {
    FG_CUDA(cudaMemsetAsync(info, 0, sizeof(int), stream));
    if (m == 0 || n == 0) return kOk;
    const int mn = m < n ? m : n;
    const size_t ws0 = getrf_workspace_bytes(m, n, tc_kind, split_nb);
    // the split GEMM's slot-0 data goes after ours; sized for the largest
    // update now so that slot 0 never moves under the panel scratch
    const size_t split_off = (ws0 + 255) / 256 * 256;
    const bool fp64_split = split_nb > 0 && tc_kind < 0;
    // look-ahead over outer blocks: its lists of row moves and the side stream's
    // operands, after ours too.  The blocks of the tensor-core LU are split_nb wide:
    // tc_buf is sized for updates of that depth.  (m bounded: panels of more than 8192
    // rows, FP32 16,384, need the whole grid and nothing runs beside them.  onb bounded
    // by the lists: a block has room for kLists panels, and the narrowest are those of
    // the whole height, half of 64 columns as a cluster's or what a grid's CTAs hold.)
    int sms = num_sms();
    if (sms <= 0) {
        set_last_error("no CUDA device");
        return kErrNoDevice;
    }
    const int gcap = panel_ctas(sms);
    const bool f32 = std::is_same<T, float>::value && panel32_enabled();   // FP32 panels, else FP64 arithmetic
    const bool cluster = !(std::is_same<T, float>::value && !f32) && cluster_fits<T>();
    // (panel_kernel holds the panel in FP64, panel32_kernel in FP32)
    const size_t panel_es = f32 ? sizeof(float) : sizeof(double);
    constexpr int kLists = 1024 / CP_NARROW, kListInts = 2 + 4 * PANEL_NB;
    int onb = !recursive ? 0 : tc_kind >= 0 ? split_nb : lookahead_nb(mn);
    const int narrowest = std::min(grid_panel_width(m, gcap, panel_es), CP_NARROW);
    if (m > 20000 || narrowest == 0 || onb > kLists * narrowest) onb = 0;
    const bool ahead_blocks = onb > 0 && mn > 2 * onb && cluster && lookahead_enabled();
    const size_t list_bytes = ((size_t)2 * kLists * kListInts * sizeof(int) + 255) / 256 * 256;
    const size_t side_bytes = tc_kind >= 0 ? tc_update_workspace_bytes(tc_kind, m, onb, PANEL_NB) : 0;
    Workspace *w = workspace_for(stream, fp64_split     ? split_off + split_ws0_bytes(m, n)
                                         : ahead_blocks ? split_off + list_bytes + side_bytes
                                                        : ws0);
    if (!w) return kErrAlloc;
    PanelScratch ps = carve_panel_scratch(w->buf);
    void *tc_buf = (char *)w->buf + (panel_scratch_bytes() + 255) / 256 * 256;
    FG_CUDA(cudaMemsetAsync(ps.slots, 0, kSlotBytes, stream));
    unsigned long long epoch = 0;
    const void *panel_fn[2] = {
        f32 ? (const void *)panel32_kernel<false> : (const void *)panel_kernel<T, false>,
        f32 ? (const void *)panel32_kernel<true> : (const void *)panel_kernel<T, true>};
    {
        static DeviceOnce once, once_d, once_f, once_fd;
        int st0 = set_smem_once(f32 ? once_f : once, panel_fn[0], (int)PANEL_SMEM_MAX);
        if (st0 == kOk) st0 = set_smem_once(f32 ? once_fd : once_d, panel_fn[1], (int)PANEL_SMEM_MAX);
        if (st0 != kOk) return st0;
    }
    // look-ahead (CUDA-core updates only: the tensor-core update is a
    // persistent kernel that leaves no SM free for a concurrent panel; with
    // its operand ring cut to 3 stages so that a panel CTA fits beside it, the
    // n = 16384 FP32 LU spent 114 ms in its updates instead of 49 and the
    // panels did not shorten)
    Workspace *wl = nullptr;
    if (tc_kind < 0 && !recursive && lookahead_enabled()) {
        wl = workspace_side(stream);
        if (!wl) return kErrCuda;
    }
    trace("getrf<%d> m=%d n=%d lda=%d panel grid<=%d update=%d lookahead=%d", (int)sizeof(T), m, n,
          ldA, gcap, tc_kind, wl ? 1 : 0);

    // columns [ob_start, ob_end) are updated by the 64-column steps
    int ob_start = 0;
    int ob_end = (split_nb > 0 && split_nb < mn) ? split_nb : n;

    // Launches the panel at column j on stream s; *jb_out = its width.
    // `defer`: overlap the panel's own rank-1 updates with its exchanges --
    // asked for when nothing large runs beside the panel.  Beside a big
    // trailing update it measured slower overall (the n = 8192 LU: 325.3
    // against 322.8 ms per solve; the GEMM took 3 ms longer, the hidden
    // panels 6 ms less), since the panel's FP64 work then competes with the
    // GEMM's on the shared SMs.
    // (FP32 storage with the FP64-arithmetic panel keeps the grid kernel)
    auto panel_at = [&](int j, cudaStream_t s, int *jb_out, bool defer, PanelScratch ps, bool beside) -> int {
        int mp = m - j;
        const int cw = cluster ? cluster_width<T>(mp, beside) : 0;
        if (cw > 0) {
            int jb = std::min(std::min(mn - j, cw), ob_end - j);
            const int R = ceil_div(mp, CP_CS);
            cudaLaunchAttribute attr;
            const cudaLaunchConfig_t cfg =
                cluster_config(&attr, (size_t)R * (jb <= CP_NARROW ? CP_NARROW : PANEL_NB) * sizeof(T), s);
            KTimer ktp(kFamPanel, s, (double)mp * jb * jb - (double)jb * jb * jb / 3.0,
                       2.0 * sizeof(T) * (double)mp * jb);
            FG_CUDA(cudaLaunchKernelEx(&cfg, panel_cluster_kernel<T>, A + j + (size_t)j * ldA, ldA, mp, jb, j,
                                       ipiv, info, w->status, ps, R));
            *jb_out = jb;
            return kOk;
        }
        int R = grid_panel_rows(mp, gcap);
        const int nb = grid_panel_width(mp, gcap, panel_es);
        if (nb == 0) {
            set_last_error("getrf: m=%d too tall for the shared-memory panel", m);
            return kErrUnsupported;
        }
        int jb = (mn - j) < nb ? (mn - j) : nb;
        if (j + jb > ob_end) jb = ob_end - j;
        const int G = ceil_div(mp, R);
        T *Ap = A + j + (size_t)j * ldA;
        int *status = w->status;
        int j0 = j;
        size_t smem = (size_t)R * jb * panel_es;
        ++epoch;
        void *args[] = {&Ap, &ldA, &mp, &jb, &j0, &ipiv, &info, &status, &ps, &R, &epoch};
        KTimer ktp(kFamPanel, s, (double)mp * jb * jb - (double)jb * jb * jb / 3.0,
                   2.0 * sizeof(T) * (double)mp * jb);
        const void *fn = panel_fn[defer ? 1 : 0];
        FG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(G),
                                            dim3(PANEL_THREADS), args, smem, s));
        *jb_out = jb;
        return kOk;
    };
    auto update_on = [&](int j, int jb, int c0, int nc, void *buf, cudaStream_t s) -> int {
        // A(j+jb:m, c0:c0+nc) -= A(j+jb:m, j:j+jb) * A(j:j+jb, c0:c0+nc)
        T *A21 = A + (j + jb) + (size_t)j * ldA;
        T *U12 = A + j + (size_t)c0 * ldA;
        T *A22 = A + (j + jb) + (size_t)c0 * ldA;
        if (tc_kind >= 0)
            return tc_trailing_update(tc_kind, m - j - jb, nc, jb, (const float *)A21, ldA,
                                      (const float *)U12, ldA, (float *)A22, ldA, buf, s);
        return gemm_tt<T>('N', 'N', m - j - jb, nc, jb, T(-1), A21, ldA, U12, ldA, T(1), A22, ldA, s);
    };
    auto update = [&](int j, int jb, int c0, int nc) -> int { return update_on(j, jb, c0, nc, tc_buf, stream); };

    // interchanges of a panel (its moves in pl) on the columns c0 .. c1 - 1 but for
    // the `skip` columns from j on
    auto interchange_on = [&](const PanelScratch &pl, int c0, int c1, int j, int skip, cudaStream_t s) -> int {
        const int ncols = c1 - c0 - skip;
        if (ncols <= 0) return kOk;
        const int blocks = ceil_div(ncols, 256 / 32);
        KTimer ktl(kFamLaswp, s, 0.0, 0.0);
        laswp_pairs_kernel<T><<<blocks, 256, 0, s>>>(A + (size_t)c0 * ldA, ldA, ncols, j - c0, skip, pl.swap_cnt,
                                                     pl.swap_dst, pl.swap_src);
        FG_CUDA(cudaGetLastError());
        return kOk;
    };
    auto interchange = [&](int j, int jb) -> int { return interchange_on(ps, 0, n, j, jb, stream); };
    auto u12_on = [&](int j, int jb, int c0, int nc, cudaStream_t s) -> int {
        return trsm_t<T>('L', 'L', 'N', 'U', jb, nc, T(1), A + j + (size_t)j * ldA, ldA, A + j + (size_t)c0 * ldA,
                         ldA, s);
    };
    // Columns j .. j + w - 1 on stream s, interchanges within [c0, c1), the moves of
    // its panels in lists[*nl], lists[*nl + 1], ...: halved, or (FP32 storage) in
    // 64-column steps as the two-level order has them.
    struct Block {
        int c0, c1, nl;
        bool beside;
        const PanelScratch *lists;              // nullptr: ps for every panel
        void *buf;
        cudaStream_t s;
    };
    auto factor = [&](auto &&self, int j, int w, Block &k) -> int {
        int st, jb = 0;
        if (w <= PANEL_NB || std::is_same<T, float>::value) {
            // (a panel of a very tall matrix comes out narrower)
            ob_end = j + w;
            if (k.lists && k.nl >= kLists) {
                set_last_error("getrf: more than %d panels in a block", kLists);
                return kErrUnsupported;
            }
            const PanelScratch &pl = k.lists ? k.lists[k.nl] : ps;
            if ((st = panel_at(j, k.s, &jb, true, pl, k.beside)) != kOk) return st;
            ++k.nl;
            if ((st = interchange_on(pl, k.c0, k.c1, j, jb, k.s)) != kOk) return st;
        } else {
            jb = ceil_div(ceil_div(w, 2), PANEL_NB) * PANEL_NB;
            if ((st = self(self, j, jb, k)) != kOk) return st;
        }
        const int c = j + jb, r = w - jb;
        if (r <= 0) return kOk;
        if ((st = u12_on(j, jb, c, r, k.s)) != kOk) return st;
        if (c < m && (st = update_on(j, jb, c, r, k.buf, k.s)) != kOk) return st;
        return self(self, c, r, k);
    };
    // Outer blocks with look-ahead: a block's panels run on 16 SMs (one cluster) and
    // wait for each other column by column, so the next block is factored on the side
    // stream while the rest of the trailing update runs beside it, on 16 SMs less
    // (kClusterSms: its persistent products would take the cluster's SMs in the gaps
    // between panels, and keep them).  Block k's interchanges on the columns outside
    // it are taken from the lists its panels left.
    if (ahead_blocks) {
        int *mem = (int *)((char *)w->buf + split_off);
        Workspace *wo = workspace_side(stream);
        if (!wo) return kErrCuda;
        {
            PanelScratch lists[2][kLists];
            for (int i = 0; i < 2 * kLists; ++i) {
                PanelScratch &q = lists[i / kLists][i % kLists];
                q = ps;
                q.swap_cnt = mem + (size_t)i * kListInts;
                q.swap_dst = q.swap_cnt + 2;
                q.swap_src = q.swap_dst + 2 * PANEL_NB;
            }
            void *side_buf = (char *)mem + list_bytes;
            cudaStream_t side = wo->side;
            bool open = false;                  // side-stream work not yet joined
            auto run = [&]() -> int {
                int st;
                Block blk[2];
                auto start = [&](int i, int j) -> int {     // block i at column j on the side stream
                    const int e = j + std::min(onb, mn - j);
                    FG_CUDA(cudaEventRecord(wo->ev_fwd, stream));
                    FG_CUDA(cudaStreamWaitEvent(side, wo->ev_fwd, 0));
                    open = true;
                    blk[i & 1] = Block{j, e, 0, true, lists[i & 1], side_buf, side};
                    const int st1 = factor(factor, j, e - j, blk[i & 1]);
                    FG_CUDA(cudaEventRecord(wo->ev_back, side));
                    return st1;
                };
                if ((st = start(0, 0)) != kOk) return st;
                for (int i = 0, j = 0; j < mn; ++i) {
                    const Block b = blk[i & 1];
                    const int e = b.c1, w = e - j;
                    FG_CUDA(cudaStreamWaitEvent(stream, wo->ev_back, 0));
                    open = false;
                    // the next block's columns (all that is left when there is none)
                    const int e2 = e < mn ? e + std::min(onb, mn - e) : n;
                    for (int l = 0; l < b.nl && e2 > e; ++l)
                        if ((st = interchange_on(b.lists[l], e, e2, e2, 0, stream)) != kOk) return st;
                    if (e2 > e) {
                        if ((st = u12_on(j, w, e, e2 - e, stream)) != kOk) return st;
                        if (e < m && (st = update_on(j, w, e, e2 - e, tc_buf, stream)) != kOk) return st;
                    }
                    if (e < mn && (st = start(i + 1, e)) != kOk) return st;
                    // the rest, beside that block's panels
                    SpareSms spare(e < mn && cluster_width<T>(m - e, true) > 0 ? kClusterSms : 0);
                    for (int l = 0; l < b.nl; ++l) {
                        if ((st = interchange_on(b.lists[l], 0, j, j, 0, stream)) != kOk) return st;
                        if ((st = interchange_on(b.lists[l], e2, n, n, 0, stream)) != kOk) return st;
                    }
                    if (n > e2) {
                        if ((st = u12_on(j, w, e2, n - e2, stream)) != kOk) return st;
                        if (e < m && (st = update_on(j, w, e2, n - e2, tc_buf, stream)) != kOk) return st;
                    }
                    j = e;
                }
                return kOk;
            };
            const int st = run();
            // never leave side-stream work unjoined, also on an error path
            if (open) cudaStreamWaitEvent(stream, wo->ev_back, 0);
            return st;
        }
    }
    if (recursive && !std::is_same<T, float>::value) {
        Block all{0, n, 0, false, nullptr, tc_buf, stream};
        const int st = factor(factor, 0, mn, all);
        if (st != kOk || n == mn) return st;
        return u12_on(0, mn, mn, n - mn, stream);
    }

    bool ahead = false;     // the panel at j was launched on the side stream
    auto body = [&]() -> int {
        int jb = 0, st;
        for (int j = 0; j < mn;) {
            if (ahead) {
                FG_CUDA(cudaStreamWaitEvent(stream, wl->ev_back, 0));
                ahead = false;
            } else if ((st = panel_at(j, stream, &jb, true, ps, false)) != kOk) {
                return st;
            }
            if ((st = interchange(j, jb)) != kOk) return st;
            int next_jb = 0;
            if (j + jb < ob_end) {
                const int nr = ob_end - j - jb;
                if ((st = trsm_t<T>('L', 'L', 'N', 'U', jb, nr, T(1), A + j + (size_t)j * ldA, ldA,
                                    A + j + (size_t)(j + jb) * ldA, ldA, stream)) != kOk)
                    return st;
                if (j + jb < m) {
                    const int nx = j + jb;
                    if (wl && nx < mn) {
                        // the next panel's columns first, then that panel on
                        // the side stream while the rest of the update runs
                        const int w2 = std::min(std::min(PANEL_NB, mn - nx), nr);
                        if ((st = update(j, jb, nx, w2)) != kOk) return st;
                        FG_CUDA(cudaEventRecord(wl->ev_fwd, stream));
                        FG_CUDA(cudaStreamWaitEvent(wl->side, wl->ev_fwd, 0));
                        // defer when the update beside the panel is small
                        // (under ~4M elements: about the panel's own time)
                        const bool small = (double)(m - j - jb) * (double)(nr - w2) < 4.0e6;
                        if ((st = panel_at(nx, wl->side, &next_jb, small, ps, false)) != kOk) return st;
                        FG_CUDA(cudaEventRecord(wl->ev_back, wl->side));
                        ahead = true;
                        if (next_jb > w2) {
                            set_last_error("getrf: look-ahead panel wider than its update");
                            return kErrUnsupported;
                        }
                        if (nr > w2 && (st = update(j, jb, nx + w2, nr - w2)) != kOk) return st;
                    } else if ((st = update(j, jb, j + jb, nr)) != kOk) {
                        return st;
                    }
                }
            }
            j += jb;
            if (ahead) jb = next_jb;
            if (j == ob_end && ob_end < n) {
                // outer block [ob_start, ob_end) done: its U12 and the trailing
                // update of everything to the right
                const int kb = ob_end - ob_start, nr = n - ob_end;
                if ((st = trsm_t<T>('L', 'L', 'N', 'U', kb, nr, T(1),
                                    A + ob_start + (size_t)ob_start * ldA, ldA,
                                    A + ob_start + (size_t)ob_end * ldA, ldA, stream)) != kOk)
                    return st;
                if (ob_end < m) {
                    st = outer_update(m - ob_end, nr, kb, A + ob_end + (size_t)ob_start * ldA, ldA,
                                      A + ob_start + (size_t)ob_end * ldA, ldA,
                                      A + ob_end + (size_t)ob_end * ldA, ldA, split_off, tc_kind,
                                      tc_buf, stream);
                    if (st != kOk) return st;
                }
                ob_start = ob_end;
                ob_end = (ob_start + split_nb < mn) ? ob_start + split_nb : n;
            }
        }
        return kOk;
    };
    const int st = body();
    // never leave side-stream work unjoined, also on an error path
    if (ahead) cudaStreamWaitEvent(stream, wl->ev_back, 0);
    return st;
}

int dgetrf_launch(int m, int n, double *A, int ldA, int *ipiv, int *info, cudaStream_t stream) {
    return getrf_t<double>(m, n, A, ldA, ipiv, info, -1, 0, stream,
                           recursive_lu(m, n, stream));
}

int dgetrf_split_launch(int m, int n, double *A, int ldA, int *ipiv, int *info, int outer_nb,
                        cudaStream_t stream) {
    if (outer_nb <= 0) outer_nb = split_outer_nb();
    if (outer_nb % PANEL_NB != 0) {
        set_last_error("dgetrf_split: outer block %d is not a multiple of %d", outer_nb, PANEL_NB);
        return kErrUnsupported;
    }
    return getrf_t<double>(m, n, A, ldA, ipiv, info, -1, outer_nb, stream);
}

int sgetrf_launch(int m, int n, float *A, int ldA, int *ipiv, int *info, int tc_kind,
                  cudaStream_t stream) {
    const int onb = tc_kind >= 0 ? tc_outer_nb() : 0;
    return getrf_t<float>(m, n, A, ldA, ipiv, info, tc_kind, onb > PANEL_NB ? onb : 0, stream,
                          onb > PANEL_NB && sgetrf_lookahead(m, n, stream));
}

template <typename T>
int getrs_t(char trans, int n, int nrhs, const T *A, int ldA, const int *ipiv, T *B, int ldB,
            cudaStream_t stream) {
    if (n == 0 || nrhs == 0) return kOk;
    int st;
    if (trans == 'N' || trans == 'n') {
        if ((st = laswp_launch_t<T>(n, nrhs, B, ldB, 1, n, ipiv, 1, stream)) != kOk) return st;
        if ((st = trsm_t<T>('L', 'L', 'N', 'U', n, nrhs, T(1), A, ldA, B, ldB, stream)) != kOk) return st;
        return trsm_t<T>('L', 'U', 'N', 'N', n, nrhs, T(1), A, ldA, B, ldB, stream);
    }
    if ((st = trsm_t<T>('L', 'U', 'T', 'N', n, nrhs, T(1), A, ldA, B, ldB, stream)) != kOk) return st;
    if ((st = trsm_t<T>('L', 'L', 'T', 'U', n, nrhs, T(1), A, ldA, B, ldB, stream)) != kOk) return st;
    return laswp_launch_t<T>(n, nrhs, B, ldB, 1, n, ipiv, -1, stream);
}

int dgetrs_launch(char trans, int n, int nrhs, const double *A, int ldA, const int *ipiv,
                  double *B, int ldB, cudaStream_t stream) {
    return getrs_t<double>(trans, n, nrhs, A, ldA, ipiv, B, ldB, stream);
}

int sgetrs_launch(char trans, int n, int nrhs, const float *A, int ldA, const int *ipiv, float *B,
                  int ldB, cudaStream_t stream) {
    return getrs_t<float>(trans, n, nrhs, A, ldA, ipiv, B, ldB, stream);
}

}  // namespace fg

// ---------------------------------------------------------------------------
// Solve without allocating: flens_gb300_dgetrs_noalloc.
//
// Some callers cannot call cudaMalloc once they are running: a service that
// reserves all of its device memory up front and must not grow it on the
// request path, code that runs inside a pre-allocated memory pool owned by
// another framework, or a host that links this library into a process where
// device allocation is forbidden after start-up (a failed or blocking
// cudaMalloc there would stall or abort the caller).  flens_gb300_dgetrs
// takes its scratch (the row permutation and gathered right-hand sides of the
// row interchanges, and for up to 4 right-hand sides the ready flags and
// status word of the chained triangular solve) from a per-stream workspace
// that it creates with cudaMalloc on first use; this entry point takes all of
// it from the fixed file-scope array below instead and calls no allocating
// routine.
//
// Limits and rules:
//  * the array holds 8 MiB: 32 KiB of chain flags, a 256-byte status word,
//    and round_up(4*n, 256) + 8*n*nrhs bytes of interchange scratch per call
//    (n = 8192 allows nrhs <= 127); larger calls are rejected with
//    FLENS_GB300_ERR_UNSUPPORTED and a message in flens_gb300_last_error();
//  * every GPU that loads the library holds the array until the process exits;
//  * all calls on a device share the one array: calls whose work overlaps on
//    the GPU (different streams, or different host threads) race on it and
//    must be serialised by the caller;
//  * the first call on a device looks the array's device address up
//    (cudaGetSymbolAddress); use inside a captured CUDA graph is not tested.
// The array keeps the last call's contents.  What must start at zero is
// cleared on the call's stream by each call (cudaMemsetAsync, which does not
// allocate): the chain flags before every chained solve, and the status
// word.  The permutation is rebuilt from the identity and the gather buffer
// is fully written before it is read.  The chained solve's waits are bounded;
// a wait that gave up (not expected: every block of that cooperative launch is
// resident) leaves its bit in the array's status word, where this entry point
// does not report it.
namespace fg {
namespace {

constexpr size_t kNoAllocScratchBytes = 8u << 20;
constexpr int kNoAllocFlags = 4096;                                   // chain flags
constexpr size_t kNoAllocHead = kNoAllocFlags * sizeof(unsigned long long) + 256;   // + status word
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

std::mutex g_noalloc_mu;
void *g_noalloc_ptr[64];

// Device address of g_noalloc_scratch on the current device, looked up once
// per device with that device current.
int noalloc_scratch(void **out) {
    int dev = -1;
    FG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_last_error("device ordinal %d out of range", dev);
        return kErrUnsupported;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || p == nullptr)
            return cuda_fail(e != cudaSuccess ? e : cudaErrorInvalidSymbol,
                             "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return kOk;
}

size_t noalloc_needed(int nrows, int ncols) {
    return ((size_t)nrows * sizeof(int) + 255) / 256 * 256 +
           (size_t)nrows * (size_t)ncols * sizeof(double);
}

// Same row interchanges as dlaswp_launch, scratch taken from `scratch`.
int laswp_fixed(int nrows, int ncols, double *A, int ldA, int k1, int k2, const int *ipiv,
                int inc, void *scratch, cudaStream_t stream) {
    if (nrows <= 0 || ncols <= 0 || k2 < k1) return kOk;
    const size_t permBytes = ((size_t)nrows * sizeof(int) + 255) / 256 * 256;
    int *perm = (int *)scratch;
    double *tmp = (double *)((char *)scratch + permBytes);
    const int use_smem = (size_t)nrows * sizeof(int) <= LASWP_SMEM ? 1 : 0;
    if (use_smem) {
        static DeviceOnce once;
        const int st0 = set_smem_once(once, (const void *)laswp_perm_kernel, LASWP_SMEM);
        if (st0 != kOk) return st0;
    }
    KTimer kt(kFamLaswp, stream, 0.0, 2.0 * (double)nrows * ncols * 16.0);
    laswp_perm_kernel<<<1, 1024, use_smem ? (size_t)nrows * sizeof(int) : 0, stream>>>(
        nrows, k1, k2, ipiv, inc, perm, use_smem);
    FG_CUDA(cudaGetLastError());
    const size_t total = (size_t)nrows * ncols;
    int blocks = (int)ceil_div(total, (size_t)256);
    if (blocks > num_sms() * 16) blocks = num_sms() * 16;
    gather_rows_kernel<double><<<blocks, 256, 0, stream>>>(nrows, ncols, A, ldA, perm, tmp);
    FG_CUDA(cudaGetLastError());
    copy_back_kernel<double><<<blocks, 256, 0, stream>>>(nrows, ncols, tmp, A, ldA);
    FG_CUDA(cudaGetLastError());
    return kOk;
}

}  // namespace
}  // namespace fg

FG_API int flens_gb300_dgetrs_noalloc(char trans, int n, int nrhs, const double *A, int ldA,
                                      const int *ipiv, double *B, int ldB, void *stream) {
    using namespace fg;
    if (trans >= 'a' && trans <= 'z') trans = (char)(trans - 'a' + 'A');
    if (trans != 'N' && trans != 'T' && trans != 'C') return -1;
    if (n < 0) return -2;
    if (nrhs < 0) return -3;
    if (ldA < (n > 1 ? n : 1)) return -5;
    if (ldB < (n > 1 ? n : 1)) return -8;
    if (n == 0 || nrhs == 0) return kOk;
    const size_t need = kNoAllocHead + noalloc_needed(n, nrhs);
    if (need > kNoAllocScratchBytes) {
        set_last_error("flens_gb300_dgetrs_noalloc: n=%d nrhs=%d needs %zu bytes of scratch, "
                       "more than its fixed %zu-byte array; use flens_gb300_dgetrs or fewer "
                       "right-hand sides per call", n, nrhs, need, kNoAllocScratchBytes);
        return kErrUnsupported;
    }
    void *base = nullptr;
    int st = noalloc_scratch(&base);
    if (st != kOk) return st;
    cudaStream_t s = (cudaStream_t)stream;
    ChainFixed fx;
    fx.flags = (unsigned long long *)base;
    fx.cap = kNoAllocFlags;
    fx.status = (int *)((char *)base + kNoAllocFlags * sizeof(unsigned long long));
    void *scratch = (char *)base + kNoAllocHead;
    FG_CUDA(cudaMemsetAsync(fx.status, 0, sizeof(int), s));
    if (trans == 'N') {
        if ((st = laswp_fixed(n, nrhs, B, ldB, 1, n, ipiv, 1, scratch, s)) != kOk) return st;
        if ((st = dtrsm_launch_fixed('L', 'L', 'N', 'U', n, nrhs, 1.0, A, ldA, B, ldB, fx, s)) != kOk)
            return st;
        return dtrsm_launch_fixed('L', 'U', 'N', 'N', n, nrhs, 1.0, A, ldA, B, ldB, fx, s);
    }
    if ((st = dtrsm_launch_fixed('L', 'U', 'T', 'N', n, nrhs, 1.0, A, ldA, B, ldB, fx, s)) != kOk)
        return st;
    if ((st = dtrsm_launch_fixed('L', 'L', 'T', 'U', n, nrhs, 1.0, A, ldA, B, ldB, fx, s)) != kOk)
        return st;
    return laswp_fixed(n, nrhs, B, ldB, 1, n, ipiv, -1, scratch, s);
}
