// mod_gemm.cu -- the FP64 GEMM on the tensor cores, by exact residues.
//
// C <- beta*C + alpha*op(A)*op(B), the large products of dgemm / syrk and of
// the LU and Cholesky updates (cxxblas/level3/gemm.tcc:42-190, syrk.tcc:42-90).
// GB300's FP64 pipe issues 2 FMAs per clock per SM (1.26 TFLOP/s); its tensor
// cores have no FP64 kind but add BF16 products of small integers exactly.
// The product is therefore formed in a residue number system (the scheme of
// Ozaki, Uchino and Imamura, "Ozaki Scheme II", 2025; the moduli are the
// largest pairwise coprime numbers up to 256, bounds and data check our own):
//
//  1. exponents: 2^e_i bounds row i of op(A), 2^f_j column j of op(B).
//  2. residues: a_ik is rounded to the integer X_ik = rint(a_ik 2^(beta-e_i)),
//     |X| <= 2^beta, and stored as its NM = 17 centred residues modulo
//     pairwise coprime p <= 256 (exact in BF16); likewise op(B).  beta is the
//     largest with 2^(2 beta) k <= P/4, P = prod p ~ 2^132, at most 61: 61 for
//     k <= 256, 59 for k = 4096 -- 6 to 8 bits more than FP64's significand.
//  3. products: one BF16 tensor-core GEMM per modulus.  |r r'| <= 2^14, so the
//     FP32 sums of 1024 products are exact integers; longer k is cut into such
//     chunks whose residues are added.  17 products where the digit form
//     (split_gemm.cu) needs 36 to 45, and every (modulus, tile) is a work item
//     of its own, so small outputs fill the GPU too.
//  4. reconstruction: X Y mod P from the residues (the operand residues of
//     op(A) already carry the inverse weights), in 160-bit integers with
//     dp4a, then ONE rounding to FP64, and C as the FP64 kernel forms it.
//
// No less accurate than FP64 arithmetic, by a check on the data: an 18th
// product of the magnitudes (rounded down to BF16) bounds Q_ij = sum_k
// |a_ik||b_kj| 2^(-e_i-f_j) from below, and their sums s_i, t_j over k are taken with
// the residues.  Rounding the operands changes c_ij by at most
// 2^(-beta-1) (s_i + t_j) 2^(e_i+f_j), s_i and t_j at most the number of nonzeros of
// column j and row i (the other entries meet zeros); a tile is accepted only if that is below
// 4 * 2^-53 * (|A||B|)_ij for all its elements with Q_ij != 0, and below 2^-53 *
// (|A||B|)_ij where the nonzeros of row i and column j do not make sure that five terms
// of the sum are nonzero.  With the rounding of the sum that is never more than FP64's
// own bound, (number of nonzero terms) * 2^-53 * (|A||B|)_ij; and a product of one
// term is exact but for that rounding, as in FP64: an entry that beta bits do not hold
// is below 2^(52-beta) of its row's range, its product with b_kj below 2^(52-beta)
// |b_kj| <= 2^(52-beta) t_j, and the second condition fails.
// Uniform entries and LU and Cholesky updates keep 4 to 6 bits
// of margin, entries u 2^e with e in [-16, 16] about one.  Tiles of data graded beyond
// that, and tiles with non-finite rows or exponents outside +-450, are left to
// the FP64 kernel, which runs last and skips all others: no readback, the
// call stays asynchronous.
#include "tcgen05.cuh"

#include <cuda_bf16.h>

#include <climits>
#include <cmath>
#include <cstdlib>

namespace fg {
namespace {

constexpr int NM = 17;                       // moduli
constexpr int NP = NM + 1;                   // operand planes: residues, magnitudes
constexpr int NG = (NM + 3) / 4;             // dp4a groups of moduli
constexpr int NL = 17;                       // base-256 limbs of P
constexpr int kPrime[NM] = {256, 255, 253, 251, 247, 241, 239, 233, 229,
                            227, 223, 217, 211, 199, 197, 193, 191};
constexpr int MT = tc::BM, NT = 256;         // output tile
constexpr int KBLK = 64;                     // k of one operand stage (128 bytes of BF16)
constexpr int CHUNK = 1024;                  // 2^14 * 1024 = 2^24: exact FP32 sums
constexpr int kExpLimit = 450;
constexpr float kMagic = 12582912.0f;        // 1.5 * 2^23: adds round to integers

struct ResConst {                            // operand side, per modulus, each value twice
    float2 p[NM], ip[NM];
    float2 ca[NM][4], cb[NM][4];             // 2^(16 t) (times the CRT inverse for A) mod p
};
struct CrtConst {
    uint32_t w[NG][NL];                      // byte l of P/p_i, four moduli per word
    uint32_t qw[NG];                         // round(2^14 / p_i)
    int P[NL];
};
struct Consts {
    ResConst res;
    CrtConst crt;
    int log2P;
};

int centred(int x, int p) {
    x %= p;
    if (x < 0) x += p;
    return 2 * x > p ? x - p : x;
}

Consts make_consts() {
    Consts c{};
    // P in base 256
    int P[NL + 1] = {1};
    for (int i = 0; i < NM; ++i) {
        int carry = 0;
        for (int l = 0; l <= NL; ++l) {
            const int v = P[l] * kPrime[i] + carry;
            P[l] = v & 255;
            carry = v >> 8;
        }
    }
    int top = NL;
    while (P[top] == 0) --top;
    c.log2P = 8 * top;
    for (int v = P[top]; v > 1; v >>= 1) ++c.log2P;
    for (int l = 0; l < NL; ++l) c.crt.P[l] = P[l];
    for (int i = 0; i < NM; ++i) {
        const int p = kPrime[i];
        int W[NL], rem = 0, wmod = 0;
        for (int l = NL - 1; l >= 0; --l) {
            const int v = rem * 256 + P[l];
            W[l] = v / p;
            rem = v % p;
        }
        for (int l = NL - 1; l >= 0; --l) wmod = (wmod * 256 + W[l]) % p;
        int y = 1;
        while ((wmod * y) % p != 1) ++y;
        for (int l = 0; l < NL; ++l) c.crt.w[i / 4][l] |= (uint32_t)W[l] << (8 * (i % 4));
        c.crt.qw[i / 4] |= (uint32_t)((2 * 16384 + p) / (2 * p)) << (8 * (i % 4));
        c.res.p[i] = make_float2(-(float)p, -(float)p);      // (negated)
        c.res.ip[i] = make_float2(1.0f / (float)p, 1.0f / (float)p);
        int b = 1;
        for (int t = 0; t < 4; ++t) {
            const float fb = (float)centred(b, p), fa = (float)centred(b * y, p);
            c.res.cb[i][t] = make_float2(fb, fb);
            c.res.ca[i][t] = make_float2(fa, fa);
            b = b * (65536 % p) % p;
        }
    }
    return c;
}
const Consts &consts() {
    static const Consts c = make_consts();
    return c;
}

// One operand as the kernels see it: R rows of op(X) along k.
struct Operand {
    const double *X;
    int ld, R, rcontig;                      // rcontig: element (r, k) at X[r + k ld], else X[k + r ld]
    unsigned *key;                           // row maxima: high word of |x|
    unsigned *sum;                           // rows: sum of the magnitudes and nonzeros (row_sum, ...)
    __nv_bfloat16 *planes;                   // NP planes of R rows x Kp
};

// The word of a row: sum of its magnitudes, rounded up to 2^-6 per 64 entries, in the low
// 19 bits, its nonzeros above them (32 bits as one atomic; 64 made every product 1.4 us
// longer).  Both hold up to 4608 entries.
constexpr unsigned kSumOne = 1u << 19;
__device__ __forceinline__ float row_sum(unsigned w) { return (float)(w & (kSumOne - 1u)) * 0.015625f; }
__device__ __forceinline__ unsigned row_nonzeros(unsigned w) { return w / kSumOne; }

// e with max|x| < 2^e from the row key; ok = false: non-finite or out of range.
__device__ __forceinline__ int key_exp(unsigned key, bool &ok) {
    const int e = (int)(key >> 20) - 1022;
    ok = key == 0u || (e >= -kExpLimit && e <= kExpLimit);
    return key == 0u ? 0 : e;
}

__device__ __forceinline__ unsigned mag_key(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
    const unsigned hi = (unsigned)(b >> 32);
    return hi ? hi : ((unsigned)b ? 1u : 0u);
}

// Every kernel here waits for the one before it before it reads or writes memory
// (griddepcontrol), so that its launch and set-up run under that one's end.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... Q>
cudaError_t launch_early(void (*fn)(P...), int grid, int block, size_t smem, cudaStream_t s, Q... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, P(args)...);
}

// ------------------------------------------------------------ exponents --
// Row maxima of |x| (as high words) by integer atomicMax into zeroed keys.
// A block takes 64 rows x 32 k (rows contiguous; 8 loads in flight per thread)
// or 8 rows x 512 k.  Bound: HBM, one read of each operand; latency when small.
constexpr int EX_K0 = 32, EX_K1 = 512;
__host__ __device__ inline int exp_blocks(int R, int K, int rcontig) {
    return rcontig ? ((R + 63) / 64) * ((K + EX_K0 - 1) / EX_K0) : ((R + 7) / 8) * ((K + EX_K1 - 1) / EX_K1);
}

__global__ void __launch_bounds__(256)
mod_exp_kernel(const __grid_constant__ Operand oa, const __grid_constant__ Operand ob, int K, int blocksA) {
    let_next_start();
    const bool isB = (int)blockIdx.x >= blocksA;
    const Operand &o = isB ? ob : oa;
    const int b = isB ? blockIdx.x - blocksA : blockIdx.x;
    if (o.rcontig) {
        __shared__ unsigned sm[4][64];
        const int rb = (o.R + 63) / 64;
        const int x = threadIdx.x & 63, y = threadIdx.x >> 6;
        const int r = (b % rb) * 64 + x, k0 = (b / rb) * EX_K0;
        unsigned m = 0u;
        if (r < o.R) {
            const double *p = o.X + (size_t)r + (size_t)k0 * o.ld;
            const int kn = min(EX_K0, K - k0);
#pragma unroll
            for (int i = 0; i < EX_K0 / 4; ++i)
                if (y + 4 * i < kn) m = max(m, mag_key(p[(size_t)(y + 4 * i) * o.ld]));
        }
        sm[y][x] = m;
        __syncthreads();
        if (y == 0 && r < o.R) {
            m = max(max(m, sm[1][x]), max(sm[2][x], sm[3][x]));
            if (m) atomicMax(&o.key[r], m);
        }
    } else {
        const int rb = (o.R + 7) / 8;
        const int lane = threadIdx.x & 31;
        const int r = (b % rb) * 8 + (threadIdx.x >> 5), k0 = (b / rb) * EX_K1;
        if (r >= o.R) return;
        const double *p = o.X + (size_t)k0 + (size_t)r * o.ld;
        const int kn = min(EX_K1, K - k0);
        unsigned m = 0u;
#pragma unroll
        for (int i = 0; i < EX_K1 / 32; ++i)
            if (lane + 32 * i < kn) m = max(m, mag_key(p[lane + 32 * i]));
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0 && m) atomicMax(&o.key[r], m);
    }
}

// ------------------------------------------------------------- residues --
// X = rint(v 2^(bits - e)) as an integer, from the bits of v.
__device__ __forceinline__ long long fixed_point(double v, int e, int bits) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    int ex = (int)((u >> 52) & 0x7FF);
    long long m = (long long)(u & 0xFFFFFFFFFFFFFull);
    if (ex) m |= 1ll << 52;
    else ex = 1;
    const int sh = ex - 1075 + bits - e;         // <= bits - 53 <= 8
    if (sh >= 0) m <<= sh;
    else if (sh > -55) m = (m + (1ll << (-sh - 1))) >> -sh;
    else m = 0;
    return (long long)u < 0 ? -m : m;
}

// |v| 2^-e rounded down to BF16's 8 significant bits; values below 2^-60 are
// raised to it, so that products of nonzeros stay nonzero in the sum.
__device__ __forceinline__ float magnitude(double v, int e) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
    if (u == 0ull) return 0.0f;
    int ex = (int)(u >> 52) - 1023 - e;          // v in [2^ex, 2^(ex+1)) 2^e
    if (ex < -60) return __uint_as_float((127u - 60u) << 23);
    const unsigned mant = (unsigned)(u >> 45) & 0x7Fu;
    return __uint_as_float(((unsigned)(ex + 127) << 23) | (mant << 16));
}

// Two FP32 operations per instruction (each lane as the scalar one).
__device__ __forceinline__ unsigned long long f2(float2 a) { return *(const unsigned long long *)&a; }
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned bf16x2(unsigned long long a) {
    unsigned d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(__uint_as_float((unsigned)(a >> 32))), "f"(__uint_as_float((unsigned)a)));
    return d;
}

// A block turns 32 rows x 64 k of one operand into its NP planes.  The tile is
// staged through shared memory so that both the FP64 reads and the BF16
// writes (16 lanes x 8 bytes = one 128-byte line per row) are coalesced; a
// thread holds 4 consecutive k, each as four signed 16-bit pieces in FP32, so
// a residue is 4 FMAs (exact: |sum| < 2^24) and 3 operations of reduction, two
// entries per instruction.  Bound: 8 bytes read and 36 written per element,
// about 60 paired FP32 instructions.
__global__ void __launch_bounds__(256, 6)
mod_residue_kernel(const __grid_constant__ Operand oa, const __grid_constant__ Operand ob, int K, int Kp,
                   int bits, int blocksA, const __grid_constant__ ResConst rc) {
    __shared__ __align__(16) double tile[32][66];
    let_next_start();
    wait_previous();
    const bool isB = (int)blockIdx.x >= blocksA;
    const Operand &o = isB ? ob : oa;
    const int b = isB ? blockIdx.x - blocksA : blockIdx.x;
    const int rb = (o.R + 31) / 32;
    const int r0 = (b % rb) * 32, k0 = (b / rb) * KBLK;
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    if (o.rcontig) {
        const int r = r0 + lane;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int k = wy + 8 * i;
            tile[lane][k] = (r < o.R && k0 + k < K) ? o.X[(size_t)r + (size_t)(k0 + k) * o.ld] : 0.0;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int rr = wy + 8 * (i >> 1), k = lane + 32 * (i & 1);
            tile[rr][k] = (r0 + rr < o.R && k0 + k < K) ? o.X[(size_t)(k0 + k) + (size_t)(r0 + rr) * o.ld] : 0.0;
        }
    }
    __syncthreads();
    const size_t plane = (size_t)o.R * Kp;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const int rr = (threadIdx.x >> 4) + 16 * h, kq = (threadIdx.x & 15) * 4;
        const int r = r0 + rr;
        if (r >= o.R) continue;
        bool ok;
        const int e = key_exp(o.key[r], ok);
        float x[4][4], mg[4];                     // [piece][entry]
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double d = ok ? tile[rr][kq + i] : 0.0;
            mg[i] = magnitude(d, e);
            long long v = fixed_point(d, e, bits);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int piece = (int)(short)(v & 0xFFFF);
                x[t][i] = (float)piece;
                v = (v - piece) >> 16;
            }
        }
        __nv_bfloat16 *out = o.planes + (size_t)r * Kp + (k0 + kq);
        // (integer sums: the same in any order; 64 entries: the sum below 2^23, their
        // number above it)
        unsigned sum = __float2uint_ru(((mg[0] + mg[1]) + (mg[2] + mg[3])) * 65536.0f);
#pragma unroll
        for (int i = 0; i < 4; ++i) sum += mg[i] != 0.0f ? 1u << 24 : 0u;
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFu << (lane & 16), sum, off);
        if ((lane & 15) == 0 && sum)
            atomicAdd(&o.sum[r], (sum >> 24) * kSumOne + (((sum & 0xFFFFFFu) + 1023u) >> 10));
        uint2 w0;
        w0.x = bf16x2(f2(make_float2(mg[0], mg[1])));
        w0.y = bf16x2(f2(make_float2(mg[2], mg[3])));
        *(uint2 *)(out + NM * plane) = w0;
        unsigned long long xl[4], xh[4];          // entries 0 and 1, 2 and 3
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            xl[t] = f2(make_float2(x[t][0], x[t][1]));
            xh[t] = f2(make_float2(x[t][2], x[t][3]));
        }
        const unsigned long long magic = f2(make_float2(kMagic, kMagic)), unmagic = f2(make_float2(-kMagic, -kMagic));
#pragma unroll
        for (int j = 0; j < NM; ++j) {
            const float2 *c = isB ? rc.cb[j] : rc.ca[j];
            const unsigned long long c0 = f2(c[0]), c1 = f2(c[1]), c2 = f2(c[2]), c3 = f2(c[3]);
            const unsigned long long ip = f2(rc.ip[j]), mp = f2(rc.p[j]);
            const unsigned long long sl = fma2(xl[3], c3, fma2(xl[2], c2, fma2(xl[1], c1, mul2(xl[0], c0))));
            const unsigned long long sh = fma2(xh[3], c3, fma2(xh[2], c2, fma2(xh[1], c1, mul2(xh[0], c0))));
            uint2 w;
            w.x = bf16x2(fma2(add2(fma2(sl, ip, magic), unmagic), mp, sl));
            w.y = bf16x2(fma2(add2(fma2(sh, ip, magic), unmagic), mp, sh));
            *(uint2 *)out = w;
            out += plane;
        }
    }
}

// ------------------------------------------------------------- products --
// Tiles of the output: all of them in bands (tc::tile_origin), or the ones
// that meet one triangle (tri 1: lower, 2: upper), column by column.
struct TileMap {
    int M, N, tm, tn, tri, ntiles;
};
TileMap make_tiles(int M, int N, int tri) {
    TileMap t{M, N, ceil_div(M, MT), ceil_div(N, NT), tri, 0};
    if (!tri) t.ntiles = t.tm * t.tn;
    for (int j = 0; tri && j < t.tn; ++j) {
        const int first = tri == 1 ? 2 * j : 0, last = tri == 1 ? t.tm : (2 * j + 2 < t.tm ? 2 * j + 2 : t.tm);
        if (last > first) t.ntiles += last - first;
    }
    return t;
}
__device__ __forceinline__ void tile_at(const TileMap &tm, int t, int &m0, int &n0) {
    if (!tm.tri) {
        tc::tile_origin(t, tm.tm, tm.tn, NT, m0, n0);
        return;
    }
    m0 = n0 = 0;
    for (int j = 0; j < tm.tn; ++j) {
        const int first = tm.tri == 1 ? 2 * j : 0;
        const int cnt = (tm.tri == 1 ? tm.tm : min(2 * j + 2, tm.tm)) - first;
        if (t < cnt) {
            m0 = (first + t) * MT;
            n0 = j * NT;
            return;
        }
        if (cnt > 0) t -= cnt;
    }
}

struct ModArgs {
    TileMap tiles;
    int nkb;                                  // 64-deep k blocks
    float qscale;                             // smallest accepted Q: this times (s_i + t_j), or 4
    unsigned dense;                           // times it: fewer nonzeros in row and column together
    uint8_t *res;                             // residues [modulus][tile][4-column group][row][4]
    uint8_t *flag;                            // per tile (row tile + tm * column tile): 1 = left to FP64
    const unsigned *keyA, *keyB;
    const unsigned *sumA, *sumB;
    float p[NM], ip[NM];
};

constexpr int STAGES = 4;
constexpr uint32_t A_BYTES = MT * 128, B_BYTES = NT * 128;
constexpr int EPI = 16;                       // epilogue warps
constexpr int MOD_THREADS = 32 * (2 + EPI);
constexpr size_t MOD_SMEM = 1024 + (size_t)STAGES * (A_BYTES + B_BYTES) + 256;

// Persistent, one CTA per SM; a work item is (plane, tile), the magnitude
// plane first.  Same roles as tc::tc_kernel (TMA producer, MMA issuer, epilogue
// warps over two TMEM accumulators), with 16 epilogue warps; a residue plane runs one
// accumulator per 1024 of k.  Epilogue: 6 FP32 operations per element reduce
// the integer sum to a centred residue, 4 are packed per word, and a warp
// stores 128 contiguous bytes per 4 columns.  MULTI (more than one chunk)
// keeps the running residue sums of the thread's 64 elements packed in 32
// registers.  Bound: the BF16 tensor pipe plus, per item, about 1.25 us that the
// accumulator's way out of TMEM adds (128 KB; 8 or 16 epilogue warps and
// prefetching the next operands into L2 measured the same): 4096 x 4096 x k takes
// 61 items of 1.25 us + 5.3 ns k per SM, 0.66 of the burst rate at k = 512, 0.89 at 4096.
template <bool MULTI>
__global__ void __launch_bounds__(MOD_THREADS, 1)
mod_product_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ ModArgs a, int *__restrict__ status) {
    using namespace tc;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem;
    uint8_t *sB = smem + STAGES * fg::A_BYTES;
    uint64_t *full = (uint64_t *)(sB + STAGES * fg::B_BYTES);
    uint64_t *empty = full + STAGES;
    uint64_t *tfull = empty + STAGES;
    uint64_t *tempty = tfull + 2;
    uint32_t *tmem_slot = (uint32_t *)(tempty + 2);
    __shared__ int s_abort;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int M = a.tiles.M, N = a.tiles.N, ntiles = a.tiles.ntiles;
    const int nitems = ntiles * NP;
    constexpr int CB = CHUNK / KBLK;             // k blocks per chunk
    const int nch = MULTI ? (a.nkb + CB - 1) / CB : 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], EPI);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    wait_previous();

    if (warp == 0) {
        if (lane == 0) {
            int q = 0, issued = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
                const int pl = it / ntiles, plane = pl == 0 ? NM : pl - 1;
                int m0, n0;
                tile_at(a.tiles, it - pl * ntiles, m0, n0);
                const int ya = plane * M + m0, yb = plane * N + n0;
                for (int k = 0; k < a.nkb; ++k, ++q) {
                    const int s = q % STAGES;
                    const uint32_t ph = (uint32_t)(q / STAGES) & 1u;
                    if (s_abort || !mbar_wait(&empty[s], ph ^ 1u, status)) {
                        s_abort = 1;
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full[s], fg::A_BYTES + fg::B_BYTES);
                    tma_load_2d(&tmA, &full[s], sA + s * fg::A_BYTES, k * KBLK, ya);
                    tma_load_2d(&tmB, &full[s], sB + s * fg::B_BYTES, k * KBLK, yb);
                    ++issued;
                }
            }
            if (!ok) {
                // let the copies already issued land before the CTA can exit
                for (int r = (issued > STAGES ? issued - STAGES : 0); r < issued; ++r)
                    mbar_wait(&full[r % STAGES], (uint32_t)(r / STAGES) & 1u, status);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = idesc_for(kTcBF16, MT, NT);
            int q = 0, i = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
                const bool mag = it < ntiles;
                const int chunks = mag ? 1 : nch;
                for (int c = 0; c < chunks && ok; ++c, ++i) {
                    const int nk = (!MULTI || mag) ? a.nkb : min(CB, a.nkb - c * CB);
                    const int b = i & 1;
                    const uint32_t acc = tmem + (uint32_t)(b * NT);
                    if (!mbar_wait(&tempty[b], ((uint32_t)(i >> 1) & 1u) ^ 1u, status)) {
                        s_abort = 1;
                        ok = false;
                        break;
                    }
                    fence_after();
                    for (int k = 0; k < nk; ++k, ++q) {
                        const int s = q % STAGES;
                        const uint32_t ph = (uint32_t)(q / STAGES) & 1u;
                        if (s_abort || !mbar_wait(&full[s], ph, status)) {
                            s_abort = 1;
                            ok = false;
                            break;
                        }
                        fence_after();
                        const uint32_t a0 = smem_u32(sA + s * fg::A_BYTES);
                        const uint32_t b0 = smem_u32(sB + s * fg::B_BYTES);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            umma<kTcBF16>(acc, sdesc_sw128(a0 + kk * 32), sdesc_sw128(b0 + kk * 32), idesc,
                                          (k | kk) != 0 ? 1u : 0u);
                        umma_commit(&empty[s]);
                    }
                    if (ok) umma_commit(&tfull[b]);
                }
            }
        }
    } else {
        const int quarter = warp & 3;                // TMEM lane quarter this warp may access
        const int cq = (warp - 2) >> 2;              // column quarter
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const int rl = quarter * 32 + lane;          // tile row
        int i = 0;
        bool live = true;
        for (int it = blockIdx.x; it < nitems && live; it += gridDim.x) {
            const int pl = it / ntiles, t = it - pl * ntiles;
            int m0, n0;
            tile_at(a.tiles, t, m0, n0);
            const bool mag = pl == 0;
            const int chunks = mag ? 1 : nch;
            const float p = mag ? 1.0f : a.p[mag ? 0 : pl - 1], ip = mag ? 1.0f : a.ip[mag ? 0 : pl - 1];
            uint8_t *out = mag ? nullptr
                               : a.res + ((size_t)(pl - 1) * ntiles + t) * (MT * NT) + (size_t)rl * 4;
            uint32_t st[MULTI ? 32 : 1];
            bool bad = false;
            unsigned wi = 0u, wj[2] = {0u, 0u};      // sums and nonzeros
            if (mag) {                               // rows' and columns' data, before the wait
                bool ok = true;
                if (m0 + rl < M) {
                    key_exp(a.keyA[m0 + rl], ok);
                    bad |= !ok;
                    wi = a.sumA[m0 + rl];
                }
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {
                    const int col = n0 + cq * 64 + cc * 32 + lane;
                    if (col < N) {
                        key_exp(a.keyB[col], ok);
                        bad |= !ok;
                        wj[cc] = a.sumB[col];
                    }
                }
            }
            for (int c = 0; c < chunks; ++c, ++i) {
                const int b = i & 1;
                if (!mbar_wait(&tfull[b], (uint32_t)(i >> 1) & 1u, status)) {
                    s_abort = 1;
                    live = false;
                    break;
                }
                fence_after();
                const uint32_t base = tmem + (uint32_t)(b * NT) + lanes;
                const bool lastc = c == chunks - 1;
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {
                    const int c0 = cq * 64 + cc * 32;
                    if (n0 + c0 >= N) break;         // uniform across the warp
                    uint32_t r[32];
                    tmem_ld32(base + (uint32_t)c0, r);
                    if (mag) {
                        // (The sparsest of the 32 columns, but for those of zeros, and the
                        // densest decide for all.  A smallest Q of -inf: no such row or column.)
                        const unsigned ni = row_nonzeros(wi), nj = row_nonzeros(wj[cc]);
                        const unsigned most = __reduce_max_sync(0xffffffffu, nj);
                        const unsigned least = __reduce_min_sync(0xffffffffu, nj ? nj : 1u << 30);
                        const float qs = ni + least >= a.dense ? a.qscale : 4.0f * a.qscale, ti = (float)ni;
                        const float pi = m0 + rl < M ? fminf(row_sum(wi), (float)most) * qs : -INFINITY;
                        const float tj = n0 + c0 + lane < N ? row_sum(wj[cc]) : -INFINITY;
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const float q = __uint_as_float(r[j]);
                            bad |= q < fmaf(fminf(__shfl_sync(0xffffffffu, tj, j), ti), qs, pi) && q != 0.0f;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const float v = __uint_as_float(r[j]);
                            const float q = fmaf(v, ip, kMagic) - kMagic;
                            float f = fmaf(-q, p, v);
                            if (!MULTI && f > 127.0f) f -= p;
                            r[j] = __float_as_uint(f + (MULTI ? kMagic + 256.0f : kMagic));
                        }
                        if (MULTI) {
                            // residues + 256 in 16-bit fields: no carries for 127 chunks
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const uint32_t w = __byte_perm(r[2 * j], r[2 * j + 1], 0x5410) & 0x03FF03FFu;
                                st[cc * 16 + j] = c == 0 ? w : st[cc * 16 + j] + w;
                            }
                            if (lastc) {
                                const float off = 256.0f * (float)chunks;
#pragma unroll
                                for (int j = 0; j < 32; ++j) {
                                    const uint32_t w = st[cc * 16 + j / 2];
                                    const float v = (float)(int)((j & 1) ? w >> 16 : w & 0xFFFFu) - off;
                                    const float q = fmaf(v, ip, kMagic) - kMagic;
                                    float f = fmaf(-q, p, v);
                                    if (f > 127.0f) f -= p;
                                    r[j] = __float_as_uint(f + kMagic);
                                }
                            }
                        }
                        if (lastc) {
#pragma unroll
                            for (int g = 0; g < 8; ++g) {
                                const uint32_t *s4 = &r[g * 4];
                                *(uint32_t *)(out + (size_t)(c0 / 4 + g) * (MT * 4)) =
                                    __byte_perm(__byte_perm(s4[0], s4[1], 0x0040), __byte_perm(s4[2], s4[3], 0x0040),
                                                0x5410);
                            }
                        }
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty[b]))
                                 : "memory");
                if (s_abort) {
                    live = false;
                    break;
                }
            }
            if (mag && __any_sync(0xffffffffu, bad) && lane == 0)
                a.flag[m0 / MT + a.tiles.tm * (n0 / NT)] = 1;
        }
    }
    // (not at the start: waiting reconstruction blocks would take the SMs left to a
    // panel on another stream)
    let_next_start();
    fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u)
                     : "memory");
    }
}

// ------------------------------------------------------- reconstruction --
__device__ __forceinline__ int dp4a_su(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// The integer sum r_i P/p_i mod P, centred, times 2^ex, rounded once (to
// nearest, ties to even) to FP64, on the integer pipe.
__device__ __forceinline__ double crt_value(const uint32_t (&g)[NG], const CrtConst &k, int ex) {
    int q = 8192;
#pragma unroll
    for (int i = 0; i < NG; ++i) q = dp4a_su(g[i], k.qw[i], q);
    q >>= 14;
    int s[NL];
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        int v = -q * k.P[l];
#pragma unroll
        for (int i = 0; i < NG; ++i) v = dp4a_su(g[i], k.w[i][l], v);
        s[l] = v;
    }
    uint32_t w[5];
    long long acc = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        acc += (long long)(s[4 * i] + (s[4 * i + 1] << 8)) + ((long long)(s[4 * i + 2] + (s[4 * i + 3] << 8)) << 16);
        w[i] = (uint32_t)acc;
        acc >>= 32;
    }
    const int top = (int)acc + s[16];
    w[4] = (uint32_t)top;
    const uint32_t neg = (uint32_t)(top >> 31);
    // magnitude: (w ^ neg) - neg
    unsigned long long c = neg & 1u;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        c += w[i] ^ neg;
        w[i] = (uint32_t)c;
        c >>= 32;
    }
    // leading word into w[4]
    int e = ex + 160;                             // value = 0.w4 w3 ... 2^e
    uint32_t sticky = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (w[4] == 0u) {
            w[4] = w[3];
            w[3] = w[2];
            w[2] = w[1];
            w[1] = w[0];
            w[0] = 0u;
            e -= 32;
        }
    }
    if (w[4] == 0u) return 0.0;
    const int z = __clz((int)w[4]);
    const uint32_t h = __funnelshift_l(w[3], w[4], z), l = __funnelshift_l(w[2], w[3], z);
    sticky = (w[2] << z) | w[1] | w[0];           // z < 32
    e -= z;
    unsigned long long m = ((unsigned long long)h << 32) | l;          // leading bit 63
    const unsigned long long rest = m & 0x7FFull;
    m >>= 11;                                     // 53 bits
    const bool up = rest > 0x400ull || (rest == 0x400ull && (sticky || (m & 1ull)));
    // e in [-900 - 122, 900 + 160]: always a normal number; the carry of the
    // rounding moves into the exponent field by itself
    const unsigned long long bits = ((unsigned long long)(e + 1021) << 52) + m + (up ? 1ull : 0ull) +
                                    ((unsigned long long)(neg & 1u) << 63);
    return __longlong_as_double((long long)bits);
}

// C from the residues.  A thread takes one row x 4 columns: its 17 residue words
// are contiguous over the warp, and C is read and written along columns, a warp
// per 256 bytes.  A block takes 8 columns of a tile (32 blocks per tile).  Bound:
// the integer pipes (about 230 operations per element, 90 of them dp4a); 17 bytes
// of residues and 16 of C move.
constexpr int CRT_PARTS = NT / 8;
__global__ void __launch_bounds__(256)
mod_crt_kernel(const __grid_constant__ TileMap tiles, const uint8_t *__restrict__ res,
               const uint8_t *__restrict__ flag, const unsigned *__restrict__ keyA,
               const unsigned *__restrict__ keyB, int bits2, double alpha, double beta,
               double *__restrict__ C, int ldC, const __grid_constant__ CrtConst k) {
    wait_previous();
    const int t = blockIdx.x / CRT_PARTS, part = blockIdx.x % CRT_PARTS;
    int m0, n0;
    tile_at(tiles, t, m0, n0);
    const int rl = threadIdx.x & 127, cg = part * 2 + (threadIdx.x >> 7);
    const int row = m0 + rl, col0 = n0 + cg * 4;
    if (row >= tiles.M || col0 >= tiles.N) return;
    if (tiles.tri == 1 && row < col0) return;
    if (tiles.tri == 2 && row > col0 + 3) return;
    const size_t tile_bytes = (size_t)MT * NT;
    const uint8_t *src = res + (size_t)t * tile_bytes + (size_t)cg * (MT * 4) + (size_t)rl * 4;
    uint32_t x[NM];
#pragma unroll
    for (int i = 0; i < NM; ++i) x[i] = __ldcs((const unsigned *)(src + (size_t)i * tiles.ntiles * tile_bytes));
    if (flag[m0 / MT + tiles.tm * (n0 / NT)]) return;     // left to the FP64 kernel
    bool ok;
    const int ea = key_exp(keyA[row], ok) - bits2;
    const bool beta1 = beta == 1.0;
    double cv[4];
    int eb[4];
    bool in[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const int col = col0 + v;
        in[v] = col < tiles.N && !(tiles.tri == 1 && row < col) && !(tiles.tri == 2 && row > col);
        cv[v] = in[v] ? C[(size_t)row + (size_t)col * ldC] : 0.0;
        eb[v] = in[v] ? key_exp(keyB[col], ok) : 0;
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        uint32_t g[NG];
#pragma unroll
        for (int i = 0; i + 3 < NM; i += 4) {
            const uint32_t lo = __byte_perm(x[i], x[i + 1], v | ((4 + v) << 4));
            const uint32_t hi = __byte_perm(x[i + 2], x[i + 3], v | ((4 + v) << 4));
            g[i / 4] = __byte_perm(lo, hi, 0x5410);
        }
        g[NG - 1] = (x[NM - 1] >> (8 * v)) & 0xFFu;
        const double s = crt_value(g, k, ea + eb[v]);
        if (in[v]) C[(size_t)row + (size_t)(col0 + v) * ldC] = fma(alpha, s, beta1 ? cv[v] : beta * cv[v]);
    }
}
static_assert(NM % 4 == 1, "the last residue group holds one modulus");

// C <- beta*C + alpha*W (tri 1/2: the lower/upper triangle), W the sum of a block's
// products over the parts of k: C is read and rounded once, as by the FP64 kernel.
__global__ void __launch_bounds__(256)
mod_finish_kernel(int m, int n, int tri, double alpha, const double *__restrict__ W, double beta,
                  double *__restrict__ C, int ldC) {
    const bool beta1 = beta == 1.0;
    const size_t total = (size_t)m * n;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(e % m), j = (int)(e / m);
        if ((tri == 1 && i < j) || (tri == 2 && i > j)) continue;
        double *c = &C[(size_t)i + (size_t)j * ldC];
        *c = fma(alpha, W[e], beta1 ? *c : beta * *c);
    }
}

size_t up256(size_t b) { return (b + 255) / 256 * 256; }

struct Layout {
    size_t keyA, keyB, sumA, sumB, flag, zeroed, planesA, planesB, res, total;
};
Layout layout_for(int m, int n, int Kp, const TileMap &t) {
    Layout l{};
    l.keyA = 0;
    l.keyB = up256((size_t)m * 4);
    l.sumA = l.keyB + up256((size_t)n * 4);
    l.sumB = l.sumA + up256((size_t)m * 4);
    l.flag = l.sumB + up256((size_t)n * 4);
    l.zeroed = l.flag + up256((size_t)t.tm * t.tn);
    l.planesA = l.zeroed;
    l.planesB = l.planesA + up256((size_t)NP * m * Kp * 2);
    l.res = l.planesB + up256((size_t)NP * n * Kp * 2);
    l.total = l.res + (size_t)NM * t.ntiles * MT * NT;
    return l;
}

// One block product at most: 1.8 GB of scratch (two operands' planes 1.4 GB, residues
// 0.3, the sum over parts of k 0.1), or 8192 x 8192 with k = 1024 (0.6 and 1.1 GB).
constexpr int kBlkK = 4608, kBlkMN = 4096;
static_assert(kBlkK * 64 < (int)kSumOne && kBlkMN <= kBlkK && kBlkK < 1 << 13, "a row's sum and nonzeros fit its word");

// One block product in the scratch `ws` (layout_for(m, n, Kp, tiles).total bytes).
int mod_block(bool ta, bool tb, int m, int n, int k, double alpha, const double *A, int ldA,
              const double *B, int ldB, double beta, double *C, int ldC, int tri, int kr, char *ws,
              int *status, cudaStream_t s) {
    const Consts &cs = consts();
    const int Kp = ceil_div(k, KBLK) * KBLK;
    const TileMap tiles = make_tiles(m, n, tri);
    const Layout l = layout_for(m, n, Kp, tiles);
    int lk = 0;
    while ((1 << lk) < k) ++lk;
    int bits = (cs.log2P - 2 - lk) / 2;
    if (bits > 61) bits = 61;
    const Operand oa{A, ldA, m, ta ? 0 : 1, (unsigned *)(ws + l.keyA), (unsigned *)(ws + l.sumA),
                     (__nv_bfloat16 *)(ws + l.planesA)};
    const Operand ob{B, ldB, n, tb ? 1 : 0, (unsigned *)(ws + l.keyB), (unsigned *)(ws + l.sumB),
                     (__nv_bfloat16 *)(ws + l.planesB)};
    FG_CUDA(cudaMemsetAsync(ws, 0, l.zeroed, s));
    {
        KTimer kt(kFamResidue, s, 0.0, 8.0 * k * ((double)m + n));
        const int ba = exp_blocks(m, k, oa.rcontig), bb = exp_blocks(n, k, ob.rcontig);
        mod_exp_kernel<<<ba + bb, 256, 0, s>>>(oa, ob, k, ba);
        FG_CUDA(cudaGetLastError());
    }
    {
        KTimer kt(kFamResidue, s, 0.0, (8.0 + 2.0 * NP) * Kp * ((double)m + n));
        const int ba = ceil_div(m, 32) * (Kp / KBLK), bb = ceil_div(n, 32) * (Kp / KBLK);
        FG_CUDA(launch_early(mod_residue_kernel, ba + bb, 256, 0, s, oa, ob, k, Kp, bits, ba, cs.res));
    }
    CUtensorMap ma, mb;
    int rc = tc::make_kmajor_map(&ma, kTcBF16, oa.planes, NP * m, Kp, Kp, MT);
    if (rc == kOk) rc = tc::make_kmajor_map(&mb, kTcBF16, ob.planes, NP * n, Kp, Kp, NT);
    if (rc != kOk) return rc;
    ModArgs a{};
    a.tiles = tiles;
    a.nkb = Kp / KBLK;
    // 2^(-bits-1) (s + t) <= 2^-51 Q; the magnitudes were rounded down by up to 2^-7
    a.qscale = (float)(1.01 * ldexp(1.0, 50 - bits));
    a.dense = k + 5;
    a.res = (uint8_t *)(ws + l.res);
    a.flag = (uint8_t *)(ws + l.flag);
    a.keyA = oa.key;
    a.keyB = ob.key;
    a.sumA = oa.sum;
    a.sumB = ob.sum;
    for (int i = 0; i < NM; ++i) {
        a.p[i] = -cs.res.p[i].x;
        a.ip[i] = cs.res.ip[i].x;
    }
    const int items = tiles.ntiles * NP, sms = num_sms() - spare_sms();
    const int grid = items < sms ? items : sms;
    {
        KTimer kt(kFamResidue, s, 2.0 * (tri ? 0.5 : 1.0) * m * (double)n * k,
                  8.0 * ((double)m * k + (double)k * n + 2.0 * m * n));
        static DeviceOnce once1, onceN;
        if (Kp <= CHUNK) {
            if ((rc = set_smem_once(once1, (const void *)mod_product_kernel<false>, (int)MOD_SMEM)) != kOk) return rc;
            FG_CUDA(launch_early(mod_product_kernel<false>, grid, MOD_THREADS, MOD_SMEM, s, ma, mb, a, status));
        } else {
            if ((rc = set_smem_once(onceN, (const void *)mod_product_kernel<true>, (int)MOD_SMEM)) != kOk) return rc;
            FG_CUDA(launch_early(mod_product_kernel<true>, grid, MOD_THREADS, MOD_SMEM, s, ma, mb, a, status));
        }
    }
    {
        KTimer kt(kFamResidue, s, 0.0, (NM + 16.0) * m * (double)n);
        FG_CUDA(launch_early(mod_crt_kernel, tiles.ntiles * CRT_PARTS, 256, 0, s, tiles, (const uint8_t *)a.res,
                             (const uint8_t *)a.flag, a.keyA, a.keyB, 2 * bits, alpha, beta, C, ldC, cs.crt));
    }
    // tiles the check refused
    return dgemm_flagged_launch(ta ? 'T' : 'N', tb ? 'T' : 'N', m, n, k, alpha, A, ldA, B, ldB, beta, C, ldC, tri,
                                a.flag, tiles.tm, kr, s);
}

int g_mode = -1;
bool mod_enabled() {
    // FLENS_GB300_DGEMM=fma|dmma selects an FP64-pipe kernel for every product
    if (g_mode < 0) {
        const char *e = getenv("FLENS_GB300_DGEMM");
        g_mode = (e && *e) ? 0 : 1;
    }
    return g_mode == 1;
}

}  // namespace

// Estimated microseconds of the two routes, fitted to measurements from 256^3 to
// 4096^3 and 1000 x 100 x 1000 to 8192 x 256 x 256 (within 15%).  FP64: an SM
// takes 0.265 us of its pipe per unit of k and 32 x 32 tile, in waves over the
// SMs.  Residues: the launches, the work items in waves (1.2 us + 5.5 ns per unit
// of k), the operands and C.  Both at, say, 300^3: 85 and 28 us; 4032 x 64 x 64: 38 and 37;
// 4096 x 128 x 128: 134 and 44.  (The FP64 kernel's 8 x 8 tiles beat that estimate: 128
// x 128 x 256 takes 26 us of a call there and 33 here, 100^3 19 and 33.  The residues
// stay: they are the more exact, and inside solves it shows.  With the smaller tiles'
// estimate LU and solve with 40 right-hand sides were 1.4 times as far off at n = 700 to
// 2500.)
bool mod_gemm_wins(int m, int n, int k, int tri, int kr) {
    if (n <= 16 || m <= 16 || k < 32 || !mod_enabled()) return false;
    const double half = tri ? 0.5 : 1.0, mn = half * m * (double)n;
    const int sms = num_sms() > 0 ? num_sms() : 1;
    const double fp64 = 5.0 + ceil(half * ceil_div(m, 32) * (double)ceil_div(n, 32) / sms) * 0.265 * k;
    const double items = ceil(half * ceil_div(m, MT) * (double)ceil_div(n, NT) * NP / sms);
    const double mod = 24.0 + items * (1.2 + 0.0055 * k) + 1.0e-5 * k * ((double)m + n) + 1.5e-5 * mn;
    // (a triangular operand has rows of few terms, whose tiles are refused: trmm 100 x 100
    // 138 us on the FP64 kernel, 160 with both; 200 x 200 236 and 184)
    return mod < (kr ? 0.75 : 0.9) * fp64;
}

// C <- beta*C + alpha*op(A)*op(B) (tri 1/2: only the lower/upper triangle of a
// square C) through residues.  kErrUnsupported when the route does not apply
// (a stream under capture, no scratch memory, or the FP64 route is faster):
// nothing has been launched then and the caller takes the FP64 kernel.
int mod_gemm_launch(char transA, char transB, int m, int n, int k, double alpha, const double *A, int ldA,
                    const double *B, int ldB, double beta, double *C, int ldC, int tri, cudaStream_t s, int kr) {
    if (!mod_gemm_wins(m, n, k, tri, kr)) return kErrUnsupported;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
        cudaGetLastError();
        return kErrUnsupported;
    }
    // its scratch would be freed while the graph still names it
    if (cap != cudaStreamCaptureStatusNone) return kErrUnsupported;
    const bool ta = !(transA == 'N' || transA == 'n'), tb = !(transB == 'N' || transB == 'n');
    // block product sizes: equal parts of at most kBlkMN x kBlkMN x kBlkK
    auto part = [](int x, int cap_, int unit) {
        const int parts = ceil_div(x, cap_);
        return ceil_div(ceil_div(x, parts), unit) * unit;
    };
    // (a triangular operand in the same parts along both its dimensions: its blocks are
    // zero, triangles, or full)
    const int kb = kr ? part(k, kBlkMN, NT) : part(k, kBlkK, KBLK);
    // a shallow product may take larger blocks of C for the same scratch
    const int capMN = !kr && kb <= 1024 ? 2 * kBlkMN : kBlkMN;
    const int mb = kr == 1 || kr == 2 ? kb : part(m, capMN, NT), nb = kr >= 3 ? kb : part(n, capMN, NT);
    const int mm = mb < m ? mb : m, nn = nb < n ? nb : n, kk = kb < k ? kb : k;
    const Layout l = layout_for(mm, nn, ceil_div(kk, KBLK) * KBLK,
                                make_tiles(mm, nn, tri && mb >= m && nb >= n ? tri : 0));
    int *status = nullptr;
    // more than one part of k: their products are summed here, then added to C
    const size_t sum_off = up256(l.total), sum_bytes = kb < k ? (size_t)mm * nn * sizeof(double) : 0;
    char *ws = (char *)scratch_acquire(sum_off + sum_bytes, s, &status);
    if (!ws) return kErrUnsupported;
    trace("dgemm: m=%d n=%d k=%d engine=residues blocks of %d x %d x %d", m, n, k, mm, nn, kk);
    double *W = sum_bytes ? (double *)(ws + sum_off) : nullptr;
    auto block = [&](int i0, int j0) -> int {
        int bt = tri;
        const int bm = m - i0 < mb ? m - i0 : mb, bn = n - j0 < nb ? n - j0 : nb;
        if (tri && i0 != j0) {
            if ((tri == 1) != (i0 > j0)) return kOk;          // the other triangle
            bt = 0;
        }
        double *Cb = C + i0 + (size_t)j0 * ldC;
        if (W) FG_CUDA(cudaMemsetAsync(W, 0, (size_t)bm * bn * sizeof(double), s));
        for (int k0 = 0; k0 < k; k0 += kb) {
            int bkr = 0;
            if (kr) {
                const int t0 = kr <= 2 ? i0 : j0;             // nonzero for k >= the row or column, else k <=
                if (kr == 1 || kr == 4 ? k0 < t0 : k0 > t0) continue;
                bkr = k0 == t0 ? kr : 0;
            }
            const int bk = k - k0 < kb ? k - k0 : kb;
            const int rc = mod_block(ta, tb, bm, bn, bk, W ? 1.0 : alpha,
                                     A + (ta ? k0 + (size_t)i0 * ldA : i0 + (size_t)k0 * ldA), ldA,
                                     B + (tb ? j0 + (size_t)k0 * ldB : k0 + (size_t)j0 * ldB), ldB, W ? 1.0 : beta,
                                     W ? W : Cb, W ? bm : ldC, bt, bkr, ws, status, s);
            if (rc != kOk) return rc;
        }
        if (W) {
            KTimer kt(kFamResidue, s, 0.0, 24.0 * bm * (double)bn);
            const size_t blocks = ((size_t)bm * bn + 255) / 256, cap = (size_t)num_sms() * 16;
            mod_finish_kernel<<<(int)(blocks < cap ? blocks : cap), 256, 0, s>>>(bm, bn, bt, alpha, W, beta, Cb, ldC);
            FG_CUDA(cudaGetLastError());
        }
        return kOk;
    };
    int rc = kOk;
    for (int i0 = 0; i0 < m && rc == kOk; i0 += mb)
        for (int j0 = 0; j0 < n && rc == kOk; j0 += nb) rc = block(i0, j0);
    scratch_release(ws, s);
    return rc;
}

}  // namespace fg
