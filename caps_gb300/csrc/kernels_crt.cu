// Residue scheme of the split base case (Ozaki scheme II: an integer modular
// technique), on tcgen05 tensor cores.
//
// The reference multiplies leaves with FP64 dgemm (multiply.cpp:1124,
// dgemm-blas.cpp:4-13).  This scheme computes the same leaf product
// C = A * B (column-major m x m, m <= 2048) as follows:
//
//  1. scale (shared with the digit scheme): per row i of A the exponent
//     bound E_i and lowest set bit, per column j of B the same; t_a, t_b =
//     min(bits needed over the launch group, 55, the cap SplitParams.bits);
//     A'_ik = round(a_ik 2^(t_a - E_i)), B'_kj = round(b_kj 2^(t_b - E_j)),
//     |A'| <= 2^t_a, |B'| <= 2^t_b, exact when the data needs <= t bits.
//  2. at the scan's end: the fewest moduli L whose product M_L exceeds
//     2 * K * 2^(t_a + t_b) (so C' = A'B' is fixed by its residues).
//  3. slice:   residues of A', B' modulo the pairwise coprime moduli
//     p_l in {181, 180, 179, 173, ...} (balanced, |r| <= 90, exact in bf16),
//     written as pre-tiled UMMA canonical K-major planes like the digits.
//  4. gemm:    per modulus, sum_k rA rB on tcgen05.mma kind::f16
//     (bf16 x bf16 -> f32): |sum| <= K 90^2 < 2^24 for K <= 2048, so the
//     fp32 accumulator is exact.  A's residues are premultiplied by
//     y_l = (M_L / p_l)^-1 mod p_l, so the sum is y_l A'B' mod p_l; drain
//     warps reduce it to its balanced residue z_l, one byte per element, in
//     a product-residue tile of the CTA.
//  5. CRT (the same warps, overlapping the next tile's MMAs): S = sum_l z_l
//     (M_L / p_l) is reduced modulo M_L and centred into (-M_L/2, M_L/2):
//     that is C' exactly; then C = C' 2^(E_i + E_j - t_a - t_b) with one
//     rounding to FP64.
//
// Against the digit scheme's 36 digit-pair products for float data, this
// takes 17 modular products for the same 55-bit operand truncation, and its
// product of the truncated operands is exact (no dropped digit pairs).
#include "split_common.cuh"

#include <cmath>

#include <cuda.h>

namespace caps {

using namespace split;

namespace {

// moduli, largest first; any prefix is pairwise coprime
__host__ __device__ constexpr int modulus(int l) {
    constexpr int m[LMAX] = {181, 180, 179, 173, 169, 167, 163, 161, 157,
                             151, 149, 139, 137, 131, 127, 121, 113};
    return m[l];
}

constexpr int RSTAGE_K = 4;                       // 16-deep K steps per stage (K = 64)
constexpr int RNSTAGE = 6;
constexpr int R_TILE = TM * TK * 2;               // 4 KiB: 128 x 16 bf16, A and B alike
constexpr int RSTAGE_OP = RSTAGE_K * R_TILE;      // 16 KiB: one operand of a stage
constexpr int RSTAGE_BYTES = 2 * RSTAGE_OP;       // 32 KiB
constexpr int MAP_ROW = 512;                      // bytes of a row of the planes' tensor map
constexpr int MAP_BOX = RSTAGE_OP / MAP_ROW;      // 32 rows: an operand's K steps of a stage
constexpr int RGEMM_THREADS = 320;                // producer, MMA, 8 drain warps
constexpr unsigned RSTATUS = 0x100;               // status bits of this kernel: RSTATUS << code

constexpr int NTRIPLE = (LMAX + 2) / 3;

struct CrtTables {
    // the slicer's constants, each in both lanes of a float2 for the packed
    // fp32 pair instructions
    float2 np2[LMAX], invp2[LMAX]; // -p_l, 1/p_l
    float2 c2[LMAX][3];            // balanced 2^(14k) mod p_l, k = 1..3
    float2 cy2[LMAX][LMAX][4];     // [L-1][l][k]: balanced 2^(14k) y_l mod p_l, k = 0..3,
                                   // y_l = (M_L / p_l)^-1 mod p_l
    // reconstruction (crt_reconstruct), per modulus count L; triple t is the
    // moduli 3t..3t+2 among the first L, P_t their product.  Limbs stand least
    // significant first.  Aligned, several constants come in one read: with
    // limbs at an offset of 12 the n = 6144 update is 0.5 % slower, with factors
    // in rows of 17 words 49 leaves of 777 at 10 moduli 1.8 %
    alignas(16) uint32_t Mt[LMAX][NTRIPLE][4];  // [L-1][t]: limbs of M_L / P_t
    alignas(16) uint32_t M[LMAX][4];            // [L-1]: limbs of M_L
    alignas(16) uint32_t Mn[LMAX][4];           // [L-1]: limbs of 2^(32 W) - M_L, W = crt_words(L)
    alignas(16) uint32_t Z0[LMAX][4];           // [L-1]: limbs of -ZOFF sum_l M_L / p_l modulo M_L
    alignas(16) uint32_t pc[LMAX][LMAX + 3];    // [L-1][l]: P_t / p_l, t = l / 3
    float m_inv[LMAX];             // [L-1]: 2^(32 (W - 2)) / M_L
};

__constant__ CrtTables c_crt;

typedef unsigned __int128 u128;

__host__ __device__ constexpr u128 moduli_product(int first, int last) {  // of the moduli first..last-1
    u128 m = 1;
    for (int l = first; l < last; l++) m *= (u128)modulus(l);
    return m;
}

// A product residue is kept balanced (|z| <= p / 2 + 1) and stored as the
// byte b = z + ZOFF, 5..187.
constexpr int ZOFF = 96, ZMAX = 187;

// 32-bit words that hold S = sum_l b_l M_L / p_l + Z0, Z0 < M_L: 2 up to 8
// moduli (M_8 < 2^59.4), 3 up to 12 (M_12 < 2^88.3), 4 up to 17 (M_17 < 2^123.1)
__host__ __device__ constexpr int crt_words(int L) { return L <= 8 ? 2 : L <= 12 ? 3 : 4; }
constexpr u128 s_bound(int L) {
    u128 v = moduli_product(0, L);
    for (int l = 0; l < L; l++) v += (u128)ZMAX * (moduli_product(0, L) / (u128)modulus(l));
    return v;
}
static_assert(s_bound(8) < ((u128)1 << 64) && s_bound(12) < ((u128)1 << 96), "S in 2 words up to L = 8, 3 up to 12");
static_assert(s_bound(LMAX) / moduli_product(0, LMAX) < 24 && moduli_product(0, LMAX) < ((u128)1 << 123) / 100 * 108,
              "S < 24 M_17 < 2^128 in 4 words");

// 32-bit limbs of M_L / P_t
__host__ __device__ constexpr int triple_limbs(int L, int t) {
    const int last = 3 * t + 3 < L ? 3 * t + 3 : L;
    u128 v = moduli_product(0, L) / moduli_product(3 * t, last);
    int n = 0;
    while (v) {
        v >>= 32;
        n++;
    }
    return n;
}

int mod_inverse(int a, int p) {
    a %= p;
    for (int x = 1; x < p; x++)
        if ((a * x) % p == 1) return x;
    return 0;
}

void build_tables(CrtTables &t) {
    for (int l = 0; l < LMAX; l++) {
        const int p = modulus(l);
        long long v = 1;
        for (int k = 1; k <= 3; k++) {
            v = (v * 16384) % p;
            long long b = v > p / 2 ? v - p : v;
            t.c2[l][k - 1] = make_float2((float)b, (float)b);
        }
        t.np2[l] = make_float2(-(float)p, -(float)p);
        t.invp2[l] = make_float2(1.0f / (float)p, 1.0f / (float)p);
    }
    for (int L = 1; L <= LMAX; L++) {
        u128 M = 1;
        for (int l = 0; l < L; l++) M *= (u128)modulus(l);
        const int W = crt_words(L);
        for (int k = 0; k < 4; k++) {
            t.M[L - 1][k] = (uint32_t)(M >> (32 * k));
            t.Mn[L - 1][k] = k < W ? (uint32_t)(((u128)0 - M) >> (32 * k)) : 0u;
        }
        u128 z0 = 0;
        for (int l = 0; l < L; l++) z0 = (z0 + (u128)(modulus(l) - ZOFF % modulus(l)) * (M / (u128)modulus(l))) % M;
        for (int k = 0; k < 4; k++) t.Z0[L - 1][k] = (uint32_t)(z0 >> (32 * k));
        t.m_inv[L - 1] = (float)(ldexp(1.0, 32 * (W - 2)) / (double)M);
        for (int i = 0; i < NTRIPLE; i++) {
            const int first = 3 * i, last = first + 3 < L ? first + 3 : L;
            const u128 P = first < L ? moduli_product(first, last) : 1;
            for (int l = first; l < last; l++) t.pc[L - 1][l] = (uint32_t)(P / (u128)modulus(l));
            for (int k = 0; k < 4; k++) t.Mt[L - 1][i][k] = first < L ? (uint32_t)((M / P) >> (32 * k)) : 0u;
        }
        for (int l = 0; l < LMAX; l++) {
            if (l >= L) {
                t.pc[L - 1][l] = 0;
                for (int k = 0; k < 4; k++) t.cy2[L - 1][l][k] = make_float2(0.f, 0.f);
                continue;
            }
            const u128 Ml = M / (u128)modulus(l);
            const int p = modulus(l), y = mod_inverse((int)(Ml % (u128)p), p);
            long long v = y;
            for (int k = 0; k < 4; k++) {
                const float b = (float)(v > p / 2 ? v - p : v);
                t.cy2[L - 1][l][k] = make_float2(b, b);
                v = (v * 16384) % p;
            }
        }
    }
}


// 1.5 * 2^23: adding it to a float of magnitude below 2^22 rounds that float
// to an integer (one rounding of the exact sum), and the low bits of the
// sum's encoding then hold the integer.  Keeps rounding and int <-> float
// conversion on the FMA pipe instead of the conversion unit.
constexpr float MAGIC = 12582912.0f;

// Residues of X = round(x 2^f) modulo the first L moduli, balanced
// (|r| <= 90).  X (|X| <= 2^55) is cut into four balanced 14-bit limbs a_k
// (X + 8192 (1 + 2^14 + 2^28 + 2^42) has ordinary base-16384 digits
// a_k + 8192; |a_k| <= 8192), or two where |X| <= 2^27; then y = sum_k a_k
// (2^(14k) mod p), balanced, has |y| < 2^21.1 and is exact in fp32, and r = y -
// p q with q = y * fl(1/p) rounded to an integer by one fused multiply-add with
// MAGIC.  That product is within |y / p| 2^-24 <= 2^-9.7 of y / p, while y / p
// lies at least 1/(2p) >= 2^-8.5 from a half-integer (or exactly on one for p =
// 180, where either neighbour gives |r| = 90), so q is a nearest integer and
// |r| <= p/2.
template <int NL>
struct Limbs {
    float a[NL];
};

// a digit 0..16384 as the float digit - 8192
__device__ __forceinline__ float balanced_digit(uint32_t d) {
    return __uint_as_float(0x4B400000u | d) - (MAGIC + 8192.0f);
}

// The limbs of X = round(x 2^f).
template <int NL>
__device__ __forceinline__ Limbs<NL> scaled_limbs14(double x, int f) {
    Limbs<NL> l;
    uint32_t ul, uh;
    if constexpr (NL == 2) {
        scaled_offset(x, f, 0x08002000u, 0u, ul, uh);  // 8192 (1 + 2^14); uh unused
        l.a[0] = balanced_digit(ul & 16383u);
        l.a[1] = balanced_digit(ul >> 14);
    } else {
        scaled_offset(x, f, 0x08002000u, 0x00800200u, ul, uh);  // 8192 sum_{k<4} 16384^k
        l.a[0] = balanced_digit(ul & 16383u);
        l.a[1] = balanced_digit((ul >> 14) & 16383u);
        l.a[2] = balanced_digit(__funnelshift_r(ul, uh, 28) & 16383u);
        l.a[3] = balanced_digit(uh >> 10);
    }
    return l;
}

// The balanced residues (|r| <= 90) of two values' integers modulo p_l, one
// per lane, on packed fp32 pair instructions: each lane performs exactly
// the scalar sequence y = a0 + a1 c0 + a2 c1 + a3 c2 (three fused
// multiply-adds, exact), q = fl(y fl(1/p) + MAGIC) - MAGIC,
// r = fl(y - q p), with round-to-nearest per lane as the scalar forms, at
// half the issued instructions.
template <int NL>
struct Limbs2 {
    float2 a[NL];  // lane x: the first value's limbs, lane y: the second's
};

template <int NL>
__device__ __forceinline__ Limbs2<NL> pair_limbs(const Limbs<NL> &u, const Limbs<NL> &v) {
    Limbs2<NL> x;
#pragma unroll
    for (int k = 0; k < NL; k++) x.a[k] = make_float2(u.a[k], v.a[k]);
    return x;
}

__device__ __forceinline__ float2 reduce_pair(float2 y, float2 invp, float2 np) {
    const float2 q = __fadd2_rn(__ffma2_rn(y, invp, make_float2(MAGIC, MAGIC)), make_float2(-MAGIC, -MAGIC));
    return __ffma2_rn(q, np, y);
}
__device__ __forceinline__ float2 reduce_pair(float2 y, int l) { return reduce_pair(y, c_crt.invp2[l], c_crt.np2[l]); }

template <int NL>
__device__ __forceinline__ float2 residue_pair(const Limbs2<NL> &x, int l) {
    const float2 *c = c_crt.c2[l];
    float2 y = __ffma2_rn(x.a[1], c[0], x.a[0]);
    if constexpr (NL == 4) y = __ffma2_rn(x.a[3], c[2], __ffma2_rn(x.a[2], c[1], y));
    return reduce_pair(y, l);
}

// the same for the integers times y_l (the CRT coefficient of modulus l among
// L): A's residues carry y_l, so each modulus's product sum is already
// y_l A'B' mod p_l, the term the CRT needs.  |y| <= 4 * 8192 * 90 < 2^21.5,
// so y / p is within 2^-9.3 of y * fl(1/p), still inside the half-integer
// margin of 2^-8.5.
template <int NL>
__device__ __forceinline__ float2 weigh_pair(const Limbs2<NL> &x, const float2 *c) {
    const float2 y = __ffma2_rn(x.a[1], c[1], __fmul2_rn(x.a[0], c[0]));
    if constexpr (NL == 4) return __ffma2_rn(x.a[3], c[3], __ffma2_rn(x.a[2], c[2], y));
    return y;
}
template <int NL>
__device__ __forceinline__ float2 residue_y_pair(const Limbs2<NL> &x, int L, int l) {
    return reduce_pair(weigh_pair(x, c_crt.cy2[L - 1][l]), l);
}

// two residues as packed bf16: |r| <= 90 has at most 7 significant bits, so
// the top half of its fp32 encoding is its exact bf16 encoding
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
}

}  // namespace

int crt_product_bits(int L) {
    const u128 M = moduli_product(0, L);
    int lg = 0;
    while ((M >> (lg + 1)) != 0) lg++;
    return lg;
}

int crt_moduli_needed(int bits, int K) {
    const int Kp = (K + TK - 1) / TK * TK;
    int kb = 0;
    while ((1 << kb) < Kp) kb++;
    for (int L = 1; L <= LMAX; L++)
        if (crt_product_bits(L) >= 2 * bits + kb + 1) return L;  // as the scan kernel: K 2^(ta+tb) < M_L / 2
    return 0;
}

// ---------------------------------------------------------------- slice
// The residues of 4 pairs of values modulo each of the first L moduli (A
// side: premultiplied by the CRT coefficients of L moduli), 8 bf16 per plane.
template <int L, int NL>
__device__ __forceinline__ void write_residues(const Limbs2<NL> (&x)[4], char *dst, size_t plane_stride, int side) {
    if (side == 0) {
#pragma unroll
        for (int l = 0; l < L; l++) {
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float2 r = residue_y_pair(x[q], L, l);
                w[q] = pack_bf16x2(r.x, r.y);
            }
            *reinterpret_cast<uint4 *>(dst + (size_t)l * plane_stride) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    } else {
#pragma unroll
        for (int l = 0; l < L; l++) {
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float2 r = residue_pair(x[q], l);
                w[q] = pack_bf16x2(r.x, r.y);
            }
            *reinterpret_cast<uint4 *>(dst + (size_t)l * plane_stride) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// The same for a modulus count known at run time, from the constants of one
// side in shared memory (a few wide loads a modulus, the same for all lanes).
// Compiled per count as well, the cases' common work was hoisted above the
// branch and spilled.
struct __align__(16) SliceConst {
    float2 c[4];  // A: 2^(14k) y_l mod p_l; B: 2^(14k) mod p_l (the first is 1)
    float2 invp, np;
};

template <int NL>
__device__ __forceinline__ void write_residues_counted(const Limbs2<NL> (&x)[4], int L, const SliceConst *consts,
                                                       char *dst, size_t plane_stride) {
#pragma unroll 1
    for (int l = 0; l < L; l++) {
        const SliceConst k = consts[l];
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float2 r = reduce_pair(weigh_pair(x[q], k.c), k.invp, k.np);
            w[q] = pack_bf16x2(r.x, r.y);
        }
        *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        dst += plane_stride;
    }
}

template <int NL>
__device__ __forceinline__ void limbs_of(const double (&v)[8], int f, Limbs2<NL> (&x)[4]) {
#pragma unroll
    for (int q = 0; q < 4; q++) x[q] = pair_limbs(scaled_limbs14<NL>(v[2 * q], f), scaled_limbs14<NL>(v[2 * q + 1], f));
}

// Residue planes, per modulus l: [l][row tile][ks] for A, [l][column tile][ks]
// for B, tiles of 128 x 16 (4 KiB), each the UMMA canonical K-major image
// (8-row x 16-byte core matrices, K halves side by side: K stride 128 B,
// row-group stride 256 B).  One thread = one row of A or column of B x 8 k, a
// block = one tile.
__device__ __forceinline__ void crt_slice_tile(const LeafTask *__restrict__ tasks, char *__restrict__ ws,
                                               const Geo &g, const SplitHdr *h, int L, int leaf, int64_t tile,
                                               int side, const SliceConst *consts) {
    const int tiles = side == 0 ? g.mtiles : 2 * g.rtiles;
    if (tile >= (int64_t)tiles * g.nks) return;
    const LeafTask t = tasks[leaf];
    const char *sc = leaf_scalars(ws, g, leaf);
    const int64_t M = g.m;
    const int tid = threadIdx.x, r = tid & 127;
    const int kg = tid >> 7;  // which 8 of the tile's 16 k
    const int64_t idx = tile / g.nks * TM + r, k0 = tile % g.nks * TK + kg * 8;
    const int64_t sk = side == 0 ? M : 1;  // stride between k
    const double *src = side == 0 ? t.A + idx + k0 * M : t.B + k0 + idx * M;
    const int ee = idx < M ? reinterpret_cast<const int *>(sc + (side == 0 ? g.off_ea : g.off_eb))[idx] : 0;
    const int tt = side == 0 ? h->ta : h->tb;
    char *dst = leaf_digits(ws, g, leaf) + (side == 0 ? g.off_ra : g.off_rb) + (size_t)tile * R_TILE +
                (size_t)(r >> 3) * 256 + (size_t)kg * 128 + (size_t)(r & 7) * 16;
    const size_t plane_stride = (size_t)tiles * g.nks * R_TILE;
    // f = t - E (ee = E + 4096; 0 for a zero row / column); padding rows,
    // columns and k give zero residues
    const bool live = idx < M && ee != 0;
    const int f = tt - (ee - 4096);
    double v[8];
    if (side == 1 && live && k0 + 8 <= M && ((uintptr_t)src & 15) == 0) {
        // a column's 8 values lie side by side: 16-byte loads
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
            const double2 w = __ldg(reinterpret_cast<const double2 *>(src + e));
            v[e] = w.x;
            v[e + 1] = w.y;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = (live && k0 + e < M) ? __ldg(src + e * sk) : 0.0;
    }
    if (L >= 15) {
        // float data need 17 moduli at 55 bits, 16 or 15 under an operand-bit
        // cap or at short K: compiled for these
        Limbs2<4> x[4];
        limbs_of(v, f, x);
        switch (L) {
            case 17: write_residues<17>(x, dst, plane_stride, side); break;
            case 16: write_residues<16>(x, dst, plane_stride, side); break;
            case 15: write_residues<15>(x, dst, plane_stride, side); break;
        }
    } else if (tt <= 27) {
        Limbs2<2> x[4];
        limbs_of(v, f, x);
        write_residues_counted(x, L, consts, dst, plane_stride);
    } else {
        Limbs2<4> x[4];
        limbs_of(v, f, x);
        write_residues_counted(x, L, consts, dst, plane_stride);
    }
}

// Grid-stride over (leaf, tile).  blockIdx.y: A (0) or B (1).  Bound by HBM at
// 17 moduli (49 leaves of 2048: 2.73 ms, 0.93 of the copy rate) and by its
// instructions at few moduli, where the limbs are most of the work: rounding
// without branches, two limbs for operands of up to 27 bits, 16-byte loads of
// B and 5 blocks an SM took 49 leaves of 1024 at 6 moduli from 508 to 364 us
// (0.83 of the copy rate), 7 leaves of 896 at 17 from 86 to 81.
__global__ void __launch_bounds__(256, 5) crt_slice_kernel(const LeafTask *__restrict__ tasks,
                                                        char *__restrict__ ws, Geo g) {
    chain_wait();
    const SplitHdr *h = reinterpret_cast<const SplitHdr *>(ws);
    const int L = h->moduli;
    __shared__ SliceConst consts[LMAX];
    if (threadIdx.x < L) {
        const int l = threadIdx.x;
        SliceConst k;
        for (int i = 0; i < 4; i++)
            k.c[i] = blockIdx.y == 0 ? c_crt.cy2[L - 1][l][i] : i == 0 ? make_float2(1.f, 1.f) : c_crt.c2[l][i - 1];
        k.invp = c_crt.invp2[l];
        k.np = c_crt.np2[l];
        consts[l] = k;
    }
    __syncthreads();
    const int64_t atiles = (int64_t)g.mtiles * g.nks, btiles = (int64_t)g.rtiles * g.nks * 2;
    const int64_t per = atiles > btiles ? atiles : btiles;
    const int64_t total = per * g.count;
    for (int64_t it = blockIdx.x; it < total; it += gridDim.x)
        crt_slice_tile(tasks, ws, g, h, L, (int)(it / per), it % per, blockIdx.y, consts);
}

// ---------------------------------------------------------------- CRT reconstruction
namespace {

// The encoding of the double nearest |v| 2^e (ties to even), with the sign
// of v, for |v| = hi 2^64 + lo < 2^127.  One rounding: the integer is rounded
// at the result's last place -- 53 significant bits, or 2^-1074 for a
// subnormal result -- and the encoding is then assembled with integer
// operations (the FP64 pipe runs at 1/64 of FP32 here): for a significand
// m <= 2^53 whose last place is 2^ex, the bits are ((ex + 1074) << 52) + m,
// which also covers subnormals (ex = -1074, m < 2^52) and a rounding carry
// into the exponent.
__device__ __forceinline__ unsigned long long round_scaled_bits(uint64_t hi, uint64_t lo, bool neg, int e) {
    if ((hi | lo) == 0) return 0;
    const int nb = hi ? 128 - __clzll((long long)hi) : 64 - __clzll((long long)lo);
    int ex = nb - 53 + e;
    if (ex < -1074) ex = -1074;
    const int s = ex - e;  // right shift of |v| that leaves the significand
    uint64_t mant;
    if (s <= 0) {
        mant = lo << (-s);  // |v| < 2^53 here
    } else if (s >= 128) {
        mant = 0;           // below half of 2^-1074
    } else {
        uint64_t q, rb, st;
        if (s < 64) {
            q = (lo >> s) | (hi << (64 - s));
            rb = (lo >> (s - 1)) & 1;
            st = lo & ((1ull << (s - 1)) - 1);
        } else if (s == 64) {
            q = hi;
            rb = lo >> 63;
            st = lo << 1;
        } else {
            q = hi >> (s - 64);
            rb = (hi >> (s - 65)) & 1;
            st = (hi & ((1ull << (s - 65)) - 1)) | lo;
        }
        mant = q + (rb & ((st != 0) | (q & 1)));
    }
    const unsigned long long sign = neg ? 0x8000000000000000ull : 0ull;
    if (ex > 971) return sign | 0x7FF0000000000000ull;  // |result| >= 2^1024
    return sign | (((unsigned long long)(ex + 1074) << 52) + mant);
}

}  // namespace

namespace {

// S += sum over the triples t = T.. of w_t (M_L / P_t), w_t = sum of the
// triple's b_l (P_t / p_l): w_t < 3 * 187 * 181 * 180 < 2^24.2, so a column sum
// of up to 6 products w_t limb stays below 2^59 and needs no carries until the end.
template <int L, int T, int W>
__device__ __forceinline__ void add_triples(const uint32_t (&z)[L], uint64_t (&s)[W]) {
    if constexpr (3 * T < L) {
        uint32_t w = z[3 * T] * c_crt.pc[L - 1][3 * T];
        if constexpr (3 * T + 1 < L) w += z[3 * T + 1] * c_crt.pc[L - 1][3 * T + 1];
        if constexpr (3 * T + 2 < L) w += z[3 * T + 2] * c_crt.pc[L - 1][3 * T + 2];
        constexpr int NL = triple_limbs(L, T);
        static_assert(NL <= W, "M_L / P_t fits the words of S");
#pragma unroll
        for (int k = 0; k < NL; k++) s[k] += (uint64_t)w * c_crt.Mt[L - 1][T][k];
        add_triples<L, T + 1, W>(z, s);
    }
}

// words of sum_k s[k] 2^(32 k) modulo 2^(32 W)
template <int W>
__device__ __forceinline__ void carry_words(const uint64_t (&s)[W], uint32_t (&w)[W]) {
    uint64_t c = s[0];
    w[0] = (uint32_t)c;
#pragma unroll
    for (int k = 1; k < W; k++) {
        c = s[k] + (c >> 32);
        w[k] = (uint32_t)c;
    }
}

// C' 2^e of one entry from its product residues' bytes b_l = z_l + ZOFF.
// S = sum_l b_l M_L / p_l + Z0 (< 2^(32 W)), congruent to sum_l z_l M_L / p_l;
// qe = S / M_L rounded, from an fp32 estimate of S's top two words (32-bit
// conversions: the 64-bit ones run on the FP64 pipe); C' = S - qe M_L, formed
// as S + qe (2^(32 W) - M_L) modulo 2^(32 W).  qe may be one off when S / M_L
// lies near a half-integer: a |C'| whose top word reaches that of M_L / 2 is
// centred exactly.  Then one rounding at the leading bit, on 32-bit words: the
// words are moved up until the top one is non-zero (for float data it is at
// once), shifted so that the top bit is bit 31, and the significand, round
// and sticky bits read off.
//
// Bound by its instructions.  Modulus products in triples and L as a template
// argument (word counts and limbs of M_L / P_t known, constants read from the
// constant bank) replace L x 4 wide multiply-adds over all 4 limbs whatever L,
// 64-bit variable shifts and a 128-bit centring per entry.  Sign and leading
// word without selects over all words where W > 2, bytes by one permute: the
// combine kernel of 7 leaves of 896 went from 55 to 50 us (244 instructions an
// entry before), the GEMM of 49 leaves of 2048 from 8.33 to 8.21 ms, of 49
// leaves of 1024 at 6 moduli from 525 to 513 us.
template <int L>
__device__ __forceinline__ unsigned long long crt_reconstruct(const uint32_t (&z)[L], int e) {
    constexpr int W = crt_words(L);
    uint64_t s[W];
#pragma unroll
    for (int k = 0; k < W; k++) s[k] = c_crt.Z0[L - 1][k];
    add_triples<L, 0, W>(z, s);
    uint32_t w[W];
    carry_words<W>(s, w);
    const float sf = fmaf((float)w[W - 1], 4294967296.0f, (float)w[W - 2]);
    const uint32_t qe = __float_as_uint(fmaf(sf, c_crt.m_inv[L - 1], MAGIC)) - 0x4B400000u;
#pragma unroll
    for (int k = 0; k < W; k++) s[k] = (uint64_t)qe * c_crt.Mn[L - 1][k] + w[k];
    carry_words<W>(s, w);
    bool neg = (w[W - 1] >> 31) != 0u;
    if constexpr (W == 2) {
        if (neg) {
            const uint64_t v = 0ull - (((uint64_t)w[1] << 32) | w[0]);
            w[0] = (uint32_t)v;
            w[1] = (uint32_t)(v >> 32);
        }
    } else {
        const uint32_t m = neg ? 0xFFFFFFFFu : 0u;
        uint64_t c = m & 1u;
#pragma unroll
        for (int k = 0; k < W; k++) {
            c += w[k] ^ m;
            w[k] = (uint32_t)c;
            c >>= 32;
        }
    }
    if constexpr (W == 2) {
        const uint64_t mag = ((uint64_t)w[1] << 32) | w[0];
        const uint64_t Mv = ((uint64_t)c_crt.M[L - 1][1] << 32) | c_crt.M[L - 1][0];
        if (mag > (Mv >> 1)) {  // C' -+ M_L has the other sign
            w[0] = (uint32_t)(Mv - mag);
            w[1] = (uint32_t)((Mv - mag) >> 32);
            neg = !neg;
        }
    } else if (w[W - 1] >= (c_crt.M[L - 1][W - 1] >> 1)) {  // |C'| perhaps above M_L / 2
        u128 mag = 0, Mv = 0;
#pragma unroll
        for (int k = 0; k < W; k++) {
            mag |= (u128)w[k] << (32 * k);
            Mv |= (u128)c_crt.M[L - 1][k] << (32 * k);
        }
        if (mag > (Mv >> 1)) {
            mag = Mv - mag;
            neg = !neg;
#pragma unroll
            for (int k = 0; k < W; k++) w[k] = (uint32_t)(mag >> (32 * k));
        }
    }
    // normalise: leading word in w[W - 1]
    int up = 0;  // words moved up
    if constexpr (W == 2) {
        up = w[1] == 0u ? 1 : 0;  // often, for integers: selects
        w[1] = up ? w[0] : w[1];
        w[0] = up ? 0u : w[0];
    } else {
#pragma unroll 1
        while (w[W - 1] == 0u && up < W - 1) {  // rarely, for float data: a branch
#pragma unroll
            for (int k = W - 1; k > 0; k--) w[k] = w[k - 1];
            w[0] = 0u;
            up++;
        }
    }
    const int lz = __clz((int)w[W - 1]);
    const int ex = 32 * (W - up) - lz - 53 + e;  // last place of a normal result
    if (w[W - 1] == 0u) return 0ull;  // a zero row or column too
    if ((unsigned)(ex + 1074) > 2045u) {
        // a result below the normal range or above the largest double
        uint64_t hi = 0, lo = 0;
        u128 mag = 0;
#pragma unroll
        for (int k = 0; k < W; k++) mag |= (u128)w[k] << (32 * k);
        mag >>= 32 * up;
        hi = (uint64_t)(mag >> 64);
        lo = (uint64_t)mag;
        return round_scaled_bits(hi, lo, neg, e);
    }
    const uint32_t th = __funnelshift_l(w[W - 2], w[W - 1], lz);  // bits 63..32 of the normalised value
    uint32_t tl, rest = 0u;                                       // bits 31..0, and whether any lie below
    if constexpr (W == 2) {
        tl = w[0] << lz;
    } else {
        tl = __funnelshift_l(w[W - 3], w[W - 2], lz);
        if constexpr (W == 3) rest = w[0] << lz;
        else rest = __funnelshift_l(w[0], w[1], lz) | (w[0] << lz);
    }
    const uint32_t ml = __funnelshift_r(tl, th, 11), mh = th >> 11;  // 53-bit significand
    const uint32_t sticky = (tl & 0x3FFu) | rest | (ml & 1u);
    const uint32_t inc = ((tl >> 10) & 1u) & (sticky ? 1u : 0u);
    const uint32_t rl = ml + inc;
    const uint32_t rh = ((uint32_t)(ex + 1074) << 20) + mh + (rl < inc ? 1u : 0u) + (neg ? 0x80000000u : 0u);
    // a carry out of the significand at the top exponent gives infinity's encoding
    return ((unsigned long long)rh << 32) | rl;
}

// A product-residue tile is eight sections, one per drain warp (its 32 rows x
// 128 columns of the unit), within each modulus's plane: word [step][lane]
// holds the bytes of columns 4 step .. 4 step + 3 of row `lane` of the section.
constexpr int ZPLANE_WORDS = TM * RTN / 4, ZSECTION_WORDS = 32 * 128 / 4, ZSTEPS = 32;

// Where a warp's section of a unit goes in C.
struct Section {
    const uint32_t *z;  // word [0][lane] of the section in modulus 0's plane
    const int *eb;      // column exponents from the section's first column on
    double *C;          // C at the lane's row and the section's first column
    int e;              // E_i - ta - tb of the lane's row, less both encodings' offsets
    int cols;           // columns of the section inside the leaf (0 or less: none)
    bool row;           // the lane's row is inside the leaf
};

template <int L>
__device__ __forceinline__ void load_step(const Section &t, int step, uint32_t (&z)[L]) {
#pragma unroll
    for (int l = 0; l < L; l++) z[l] = t.z[l * ZPLANE_WORDS + step * 32];
}

// C of one step: four columns of the lane's row
template <int L>
__device__ __forceinline__ void reconstruct_step(const Section &t, int step, const uint32_t (&zq)[L], int64_t M) {
    double *dst = t.C + (int64_t)(4 * step) * M;
    // one entry at a time: unrolled by 2 or 4 it ran no faster (two warps per
    // scheduler cover the latencies) and spilled registers
#pragma unroll 1
    for (int q = 0; q < 4 && 4 * step + q < t.cols; q++) {
        uint32_t z[L];
#pragma unroll
        for (int l = 0; l < L; l++) z[l] = __byte_perm(zq[l], 0u, 0x4440u + q);  // byte q
        // C = C' 2^(E_i + E_j - ta - tb); a zero row / column has C' = 0
        const unsigned long long v = crt_reconstruct<L>(z, t.e + t.eb[4 * step + q]);
        if (t.row) dst[q * M] = __longlong_as_double((long long)v);
    }
}

}  // namespace

// ---------------------------------------------------------------- gemm
// Persistent, one CTA per SM in pairs (clusters of two), 320 threads: warp 0
// loads (one lane, TMA boxes of pre-tiled planes), warp 1 issues the MMAs (one
// lane of the pair's first CTA), warps 2..9 drain the accumulators and
// reconstruct C.
//
// A work unit is (leaf, two 128-row tiles, 256-column tile).  For each modulus
// in turn it takes Kp / 16 MMAs of 256 x 256 x 16 on both SMs: a CTA loads its
// own 128 rows of A and half of the columns of B, and its 128 x 256 results
// fall into one of two TMEM accumulators of its own; they alternate, so the
// drain of one modulus overlaps the MMAs of the next.  Against one-CTA MMAs of
// 128 x 256 x 16 an SM loads and reads 8 KiB per MMA instead of 12, and six
// stages of K = 64 fit instead of four: that kernel's issuer waited for data a
// third of the time.  49 leaves of 2048 at 17 moduli: 10.2 -> 8.53 ms (1405 ->
// 1677 TFLOP/s of modular products); 49 leaves of 1536: 4.53 -> 3.80 ms (ncu;
// the one-CTA kernel with its own reconstruction warps).  A last odd row tile
// leaves the second CTA's half unused.
// The drain reduces each exact sum modulo p (two values per packed fp32
// instruction) and stores the balanced residue as a byte, four columns to a
// word, into its section of the CTA's product-residue tile; two tiles per CTA
// are used in turn.
//
// A drain warp also reconstructs the section it drained for the unit before:
// ceil(32 / L) steps of 32 rows x 4 columns after each modulus's drain.  The
// words of a step are loaded one modulus ahead, so their way through L2 and
// DRAM (two tiles per CTA exceed L2) runs beside the wait for the accumulator
// and the drain.  Four warps of their own, one column ahead, were bound by
// that latency: 4000 clocks per 128 entries at L = 17 and 2900 at L = 6, that
// is 256 k clocks a unit beside 278 k (K = 2048, L = 17) or 49 k (K = 1024,
// L = 6) of MMAs.  A section is written and read by one warp, so no barrier
// hands tiles over.  Measured against those four warps (us a multiply): the
// n = 16384 integer case (L = 6, leaves of 1024) 139400 -> 102300, n = 6144
// (leaves of 1536) 7780 -> 7445, one leaf of 448 294 -> 205 (one-CTA MMAs).
//
// Units are ordered leaf, row tiles, column tile, and the CTAs go through the
// moduli in step, so the CTAs running at one time share the A and B planes
// of one modulus of about one leaf (16 MB at m = 2048) through L2.
//
// That needs many units a pair.  A launch with few of them (one leaf of 448
// has 4, for 76 pairs) hands out (unit, modulus) items instead, in turn, all
// units of a modulus before the next, so that the pairs still share its planes
// (as runs of one unit's moduli, a leaf of 1792 read every tile's planes from
// DRAM: 210 us instead of 111).  Each unit then has a residue tile per CTA, and
// crt_combine_kernel turns the tiles into C with the whole GPU;
// launch_crt_gemm_leaves and launch_crt_gemm have the rules.
struct Items {
    uint32_t total, pairs, c, L, count;
    int split;

    __device__ Items(int64_t units, int L_, int split_) : split(split_) {
        total = (uint32_t)units;
        L = (uint32_t)L_;
        c = blockIdx.x >> 1;
        pairs = gridDim.x >> 1;
        const uint32_t n = split ? total * L : total;  // items or units handed out in turn
        count = c < n ? (n - c + pairs - 1) / pairs : 0;
        if (!split) count *= L;
    }
    // this pair's k-th item: unit u, modulus l
    __device__ void get(uint32_t k, uint32_t &u, uint32_t &l) const {
        if (split) {
            const uint32_t i = c + k * pairs;
            l = i / total;
            u = i - l * total;
        } else {
            const uint32_t i = k / L;
            l = k - i * L;
            u = c + i * pairs;
        }
    }
};

struct DrainArgs {
    const LeafTask *tasks;
    char *ws;
    const Geo *g;
    unsigned char *ztiles;
    unsigned *status;
    uint32_t tmem, tfull0, tempty0, wl;  // tempty0: the leader's, a shared::cluster address
    uint32_t rank;                       // of this CTA in its pair
    int64_t total;
    int tab;
};

// One accumulator's residues into a warp's section of modulus l's plane; the
// accumulator is free afterwards.
__device__ __forceinline__ void drain_modulus(const DrainArgs &a, int l, uint32_t acc, int quarter, int colhalf,
                                              uint32_t *out) {
    tc_fence_after();
    const float2 invp = c_crt.invp2[l], np = c_crt.np2[l];
#pragma unroll 1
    for (int c4 = 0; c4 < 4; c4++) {
        uint32_t v[32];
        tmem_ld32(a.tmem + ((uint32_t)(quarter * 32) << 16) + acc * RTN + colhalf * 128 + c4 * 32, v);
#pragma unroll
        for (int w = 0; w < 8; w++) {
            // c = sum rA rB = y A'B' mod p (exact, |c| < 2^24; A's residues
            // carry y).  q = c fl(1/p) rounded by MAGIC is within 1/2 +
            // |c / p| 2^-24 <= 1/2 + 1/p of c / p, so z = c - q p has |z| <=
            // p / 2 + 1 and z = c mod p.
            uint32_t b[4];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float2 c = make_float2(__uint_as_float(v[4 * w + 2 * h]), __uint_as_float(v[4 * w + 2 * h + 1]));
                const float2 q =
                    __fadd2_rn(__ffma2_rn(c, invp, make_float2(MAGIC, MAGIC)), make_float2(-MAGIC, -MAGIC));
                const float2 z = __fadd2_rn(__ffma2_rn(q, np, c), make_float2(MAGIC + ZOFF, MAGIC + ZOFF));
                b[2 * h] = __float_as_uint(z.x);  // low byte: z + ZOFF
                b[2 * h + 1] = __float_as_uint(z.y);
            }
            out[(c4 * 8 + w) * 32] =
                __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
        }
    }
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive_remote(a.tempty0 + 8 * acc);
}

// A warp's section of unit u, tile row and column offsets of the section given.
__device__ __forceinline__ Section unit_section(const LeafTask *__restrict__ tasks, char *__restrict__ ws,
                                                const Geo &g, int tab, int64_t u, int rank, int section,
                                                const uint32_t *z) {
    const int64_t M = g.m, tiles = (int64_t)((g.mtiles + 1) / 2) * g.rtiles, tile = u % tiles;
    const int leafi = (int)(u / tiles), lane = threadIdx.x & 31;
    // sections are numbered by drain warp: warp 2 + section has TMEM quarter (2 + section) % 4
    const int quarter = (2 + section) & 3, colhalf = section >> 2;
    const int mt = 2 * (int)(tile / g.rtiles) + rank, rt = (int)(tile % g.rtiles);
    const char *sc = leaf_scalars(ws, g, leafi);
    const int64_t i = (int64_t)mt * TM + quarter * 32 + lane, j = (int64_t)rt * RTN + colhalf * 128;
    Section t;
    t.row = i < M;
    t.e = (t.row ? reinterpret_cast<const int *>(sc + g.off_ea)[i] : 0) - 8192 - tab;
    t.eb = reinterpret_cast<const int *>(sc + g.off_eb) + j;
    t.z = z;
    t.C = tasks[leafi].C + i + j * M;
    t.cols = mt >= g.mtiles ? 0 : (int)(M - j < 128 ? M - j : 128);
    return t;
}

// split launches: the residues alone, each unit's into a tile of its own
__device__ __forceinline__ void drain_only(const DrainArgs &a, const Items &items) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quarter = warp & 3, colhalf = (warp - 2) >> 2;
    for (uint32_t k = 0; k < items.count; k++) {
        uint32_t u, l;
        items.get(k, u, l);
        const bool got = mbar_wait(a.tfull0 + 8 * (k & 1), (k >> 1) & 1, a.status, RSTATUS << 5, a.wl);
        if (!__all_sync(0xffffffffu, got)) return;
        drain_modulus(a, (int)l, k & 1, quarter, colhalf,
                      reinterpret_cast<uint32_t *>(a.ztiles + (size_t)(2 * u + a.rank) * ZTILE_BYTES) +
                          (size_t)l * ZPLANE_WORDS + (warp - 2) * ZSECTION_WORDS + lane);
    }
}

template <int L>
__device__ __forceinline__ void drain_and_reconstruct(const DrainArgs &a) {
    constexpr int NC = (ZSTEPS + L - 1) / L;        // reconstruction steps per modulus
    constexpr int NB = NC * L <= 40 ? NC : 40 / L;  // steps held in registers at a time
    const Geo &g = *a.g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quarter = warp & 3;         // TMEM lanes 32*quarter.. (rows of the tile)
    const int colhalf = (warp - 2) >> 2;  // columns 128*colhalf.. of the tile
    const int64_t M = g.m;
    uint32_t uc = 0, tc = 0;
    Section prev;
    prev.cols = 0;
    bool have = false;
    // one more pass than units: the last unit's reconstruction
    for (int64_t u = blockIdx.x >> 1;; u += gridDim.x >> 1, tc++) {
        const bool live = u < a.total;
        if (!live && !have) return;
        uint32_t *zt = reinterpret_cast<uint32_t *>(a.ztiles + (size_t)(tc & 1) * ZTILE_BYTES) +
                       (warp - 2) * ZSECTION_WORDS + lane;
        uint32_t zr[NB][L], zn[NB][L];
        auto load = [&](int first, uint32_t (&z)[NB][L]) {
#pragma unroll
            for (int b = 0; b < NB; b++)
                if (4 * (first + b) < prev.cols) load_step<L>(prev, first + b, z[b]);
        };
        load(0, zr);
#pragma unroll 1
        for (int l = 0; l < L; l++) {
            const int s0 = l * NC, s1 = s0 + NC < ZSTEPS ? s0 + NC : ZSTEPS;
            if (s0 + NC < ZSTEPS) load(s0 + NC, zn);  // for the next modulus
            if (live) {
                const uint32_t acc = uc & 1;
                // warp-uniform: tcgen05.ld below is .sync.aligned
                const bool got = mbar_wait(a.tfull0 + 8 * acc, (uc >> 1) & 1, a.status, RSTATUS << 5, a.wl);
                if (!__all_sync(0xffffffffu, got)) return;
                drain_modulus(a, l, acc, quarter, colhalf, zt + (size_t)l * ZPLANE_WORDS);
                uc++;
            }
#pragma unroll 1
            for (int s = s0; s < s1; s += NB) {
                if (s != s0) load(s, zr);
#pragma unroll
                for (int b = 0; b < NB; b++)
                    if (s + b < s1 && 4 * (s + b) < prev.cols) reconstruct_step<L>(prev, s + b, zr[b], M);
            }
#pragma unroll
            for (int b = 0; b < NB; b++)
#pragma unroll
                for (int k = 0; k < L; k++) zr[b][k] = zn[b][k];
        }
        if (!live) return;
        __syncwarp();  // the section's words, written by all lanes, are read from here on
        prev = unit_section(a.tasks, a.ws, g, a.tab, u, (int)a.rank, warp - 2, zt);
        have = true;
    }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(RGEMM_THREADS, 1)
    crt_gemm_kernel(const LeafTask *__restrict__ tasks, char *__restrict__ ws, Geo g,
                    const __grid_constant__ CUtensorMap planes, unsigned *__restrict__ status, int split,
                    int starve) {
    // starve (test hook): no copies are issued, so nothing is ever in flight
    // and every wait may give up after a short spin
    const uint32_t wl = starve ? WAIT_LIMIT_STARVED : WAIT_LIMIT;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *stA = smem;                        // RNSTAGE x RSTAGE_OP
    unsigned char *stB = smem + RNSTAGE * RSTAGE_OP;  // RNSTAGE x RSTAGE_OP
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + RNSTAGE * RSTAGE_BYTES);
    // bars: full[RNSTAGE] (the leader's count both CTAs' copies), empty[RNSTAGE]
    // and tfull[2] (each CTA's, from the leader's commits), tempty[2] (the
    // leader's, from both CTAs' drain warps), final
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * RNSTAGE + 5);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + RNSTAGE);
    const uint32_t tfull0 = smem_u32(bars + 2 * RNSTAGE), tempty0 = smem_u32(bars + 2 * RNSTAGE + 2);
    const uint32_t finalb = smem_u32(bars + 2 * RNSTAGE + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();

    if (threadIdx.x == 0) {
        for (int i = 0; i < RNSTAGE; i++) {
            mbar_init(full0 + 8 * i, 1);
            mbar_init(empty0 + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(tfull0 + 8 * i, 1);
            mbar_init(tempty0 + 8 * i, 16);  // the 8 drain warps of both CTAs
        }
        mbar_init(finalb, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                         smem_u32(tmem_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    chain_wait();
    const SplitHdr *h = reinterpret_cast<const SplitHdr *>(ws);
    const int L = h->moduli;

    const int64_t tiles = (int64_t)((g.mtiles + 1) / 2) * g.rtiles;
    const int64_t total = tiles * g.count;
    const int nks = g.nks;
    const Items items(total, L, split);
    unsigned char *ztiles = (unsigned char *)ws + g.z_base + (split ? 0 : (size_t)blockIdx.x * 2 * ZTILE_BYTES);

    if (warp == 0) {
        // ------------------------------------------------ producer (both CTAs)
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            uint32_t armed[RNSTAGE];  // 1 + phase of the last arm
            for (int i = 0; i < RNSTAGE; i++) armed[i] = 0;
            const uint32_t lead_full = map_to_rank(full0, 0);
            for (uint32_t k = 0; k < items.count && ok && !starve; k++) {
                uint32_t u, l;
                items.get(k, u, l);
                const uint32_t leafi = u / (uint32_t)tiles, tile = u - leafi * (uint32_t)tiles;
                int mt = 2 * (int)(tile / g.rtiles) + (int)rank;
                if (mt >= g.mtiles) mt = g.mtiles - 1;  // results unused
                const int ct = 2 * (int)(tile % g.rtiles) + (int)rank;
                const size_t pl = (size_t)leafi * g.dg_per_leaf;
                // rows of the tensor map; a box past the tile's last K step
                // brings what follows it (zeros at the map's end), unused
                const int rowA = (int)((pl + g.off_ra + ((size_t)l * g.mtiles + mt) * nks * R_TILE) / MAP_ROW);
                const int rowB = (int)((pl + g.off_rb + ((size_t)l * 2 * g.rtiles + ct) * nks * R_TILE) / MAP_ROW);
                for (int ks = 0; ks < nks; ks += RSTAGE_K) {
                    if (!mbar_wait(empty0 + 8 * stage, phase ^ 1, status, RSTATUS << 0, wl)) { ok = false; break; }
                    if (rank == 0) mbar_expect_tx(full0 + 8 * stage, 2 * RSTAGE_BYTES);
                    tma_row_box_pair(smem_u32(stA + stage * RSTAGE_OP), &planes, rowA + ks * (R_TILE / MAP_ROW),
                                     lead_full + 8 * stage);
                    tma_row_box_pair(smem_u32(stB + stage * RSTAGE_OP), &planes, rowB + ks * (R_TILE / MAP_ROW),
                                     lead_full + 8 * stage);
                    armed[stage] = 1 + phase;
                    if (++stage == RNSTAGE) { stage = 0; phase ^= 1; }
                }
            }
            // every armed stage's copies, both CTAs', land before either exits
            for (int i = 0; i < RNSTAGE; i++)
                if (rank == 0 && armed[i]) mbar_wait(full0 + 8 * i, armed[i] - 1, status, RSTATUS << 1, wl);
            // and so have the leader's commits on this CTA's barriers
            for (int i = 0; i < RNSTAGE && ok; i++)
                if (armed[i]) ok = mbar_wait(empty0 + 8 * i, armed[i] - 1, status, RSTATUS << 0, wl);
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer (the leader)
        if (rank == 0 && lane == 0) {
            // K-direction core-matrix stride (LBO) 128 B, row-group stride (SBO) 256 B
            const uint64_t a0 = sdesc(smem_u32(stA), 128, 256), b0 = sdesc(smem_u32(stB), 128, 256);
            const uint32_t idesc = idesc_bf16(2 * TM, RTN);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (uint32_t k = 0; k < items.count && ok; k++) {
                const uint32_t acc = k & 1;
                if (!mbar_wait(tempty0 + 8 * acc, ((k >> 1) & 1) ^ 1, status, RSTATUS << 2, wl)) break;
                tc_fence_after();
                const uint32_t dt = tmem + acc * RTN;
                for (int ks = 0; ks < nks; ks += RSTAGE_K) {
                    const int n = ks + RSTAGE_K <= nks ? RSTAGE_K : nks - ks;
                    if (!mbar_wait(full0 + 8 * stage, phase, status, RSTATUS << 3, wl)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t so = (uint64_t)((uint32_t)stage * RSTAGE_OP) >> 4;
#pragma unroll
                    for (int j = 0; j < RSTAGE_K; j++)
                        if (j < n)
                            umma_pair(dt, a0 + so + (uint64_t)(j * R_TILE >> 4), b0 + so + (uint64_t)(j * R_TILE >> 4),
                                      idesc, (ks + j) > 0 ? 1u : 0u);
                    umma_commit_pair(empty0 + 8 * stage);
                    if (++stage == RNSTAGE) { stage = 0; phase ^= 1; }
                }
                if (ok) umma_commit_pair(tfull0 + 8 * acc);
            }
            // every issued MMA completes before TMEM is released
            umma_commit_pair_local(finalb);
            mbar_wait(finalb, 0, status, RSTATUS << 4, wl);
        }
    } else {
        // ------------------------------------------------ drain and reconstruction (8 warps)
        const DrainArgs a{tasks,  ws,     &g, ztiles, status, tmem, tfull0, map_to_rank(tempty0, 0),
                          wl,     rank,   total, h->ta + h->tb};
        if (split) drain_only(a, items);
        else switch (L) {
#define CAPS_DRAIN(n) case n: drain_and_reconstruct<n>(a); break;
            CAPS_DRAIN(1) CAPS_DRAIN(2) CAPS_DRAIN(3) CAPS_DRAIN(4) CAPS_DRAIN(5) CAPS_DRAIN(6)
            CAPS_DRAIN(7) CAPS_DRAIN(8) CAPS_DRAIN(9) CAPS_DRAIN(10) CAPS_DRAIN(11) CAPS_DRAIN(12)
            CAPS_DRAIN(13) CAPS_DRAIN(14) CAPS_DRAIN(15) CAPS_DRAIN(16) CAPS_DRAIN(17)
#undef CAPS_DRAIN
        }
        static_assert(LMAX == 17, "every modulus count is covered");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // neither CTA leaves while the other may read its shared memory or arrive on its barriers
    tc_fence_after();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// ---------------------------------------------------------------- combine
// C from the residue tiles of a split launch: a warp per step of a section
// (32 rows x 4 columns), blockIdx.x over (tile, section, four steps).  Its
// loads are independent and its arithmetic is that of the drain warps; with
// every SM at it one leaf of 448 takes 8 us and one of 2048 41; the GEMM kernel
// of the leaf of 448 took 111 us with its 4 pairs reconstructing, and takes 11.
template <int L>
__device__ __forceinline__ void combine_step(const Section &t, int step, int64_t M) {
    uint32_t z[L];
    load_step<L>(t, step, z);
    reconstruct_step<L>(t, step, z, M);
}

__global__ void __launch_bounds__(128) crt_combine_kernel(const LeafTask *__restrict__ tasks, char *__restrict__ ws,
                                                          Geo g) {
    chain_wait();
    const SplitHdr *h = reinterpret_cast<const SplitHdr *>(ws);
    const int section = (blockIdx.x >> 3) & 7, step = (blockIdx.x & 7) * 4 + (threadIdx.x >> 5);
    const int64_t tile = blockIdx.x >> 6;
    const uint32_t *z = reinterpret_cast<const uint32_t *>(ws + g.z_base + (size_t)tile * ZTILE_BYTES) +
                        section * ZSECTION_WORDS + (threadIdx.x & 31);
    const Section t = unit_section(tasks, ws, g, h->ta + h->tb, tile >> 1, (int)(tile & 1), section, z);
    if (4 * step >= t.cols) return;
    switch (h->moduli) {
#define CAPS_COMBINE(n) case n: combine_step<n>(t, step, g.m); break;
        CAPS_COMBINE(1) CAPS_COMBINE(2) CAPS_COMBINE(3) CAPS_COMBINE(4) CAPS_COMBINE(5) CAPS_COMBINE(6)
        CAPS_COMBINE(7) CAPS_COMBINE(8) CAPS_COMBINE(9) CAPS_COMBINE(10) CAPS_COMBINE(11) CAPS_COMBINE(12)
        CAPS_COMBINE(13) CAPS_COMBINE(14) CAPS_COMBINE(15) CAPS_COMBINE(16) CAPS_COMBINE(17)
#undef CAPS_COMBINE
    }
}

// ---------------------------------------------------------------- launchers
static CrtTables g_tables_host;
static bool g_tables_built = false;
static int g_crt_device = -1;
static cudaError_t g_crt_error = cudaSuccess;
static decltype(&cuTensorMapEncodeTiled) g_encode_tiled = nullptr;

cudaError_t crt_prepare() {
    int dev = 0;
    cudaGetDevice(&dev);
    if (g_crt_device == dev) return g_crt_error;
    if (!g_tables_built) {
        build_tables(g_tables_host);
        g_tables_built = true;
    }
    g_crt_error = cudaMemcpyToSymbol(c_crt, &g_tables_host, sizeof(CrtTables));
    if (g_crt_error == cudaSuccess) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        g_crt_error = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found);
        if (g_crt_error == cudaSuccess && (found != cudaDriverEntryPointSuccess || !fn)) g_crt_error = cudaErrorNotSupported;
        g_encode_tiled = (decltype(&cuTensorMapEncodeTiled))fn;
    }
    if (g_crt_error == cudaSuccess) {
        const size_t smem = (size_t)RNSTAGE * RSTAGE_BYTES + 1024 + 1024;
        g_crt_error = cudaFuncSetAttribute(crt_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
    g_crt_device = dev;
    return g_crt_error;
}

cudaError_t launch_crt_slice(const LeafTask *tasks_dev, int count, int m, SplitParams p, void *workspace,
                             cudaStream_t stream) {
    // the moduli tables must be on the device before the first launch group
    // of the process (returns at once afterwards)
    cudaError_t e = crt_prepare();
    if (e != cudaSuccess) return e;
    Geo g = make_geo(m, count, p.scheme);
    const int64_t atiles = (int64_t)g.mtiles * g.nks, btiles = (int64_t)g.rtiles * g.nks * 2;
    const int64_t items = (atiles > btiles ? atiles : btiles) * count;
    dim3 grid((unsigned)(items < 4096 ? items : 4096), 2);
    count_launch();
    return launch_chained(crt_slice_kernel, grid, 256, 0, stream, tasks_dev, (char *)workspace, g);
}

// units of a leaf: two row tiles by a column tile
static int64_t leaf_units(const Geo &g) { return (int64_t)((g.mtiles + 1) / 2) * g.rtiles; }

// One GEMM launch over g.count leaves, and the combine kernel after it for items.
static cudaError_t launch_crt_gemm_leaves(const LeafTask *tasks_dev, char *ws, const Geo &g, unsigned int *status_dev,
                                          int num_sms, cudaStream_t stream, int starve) {
    // the leaves' plane blocks as rows of 512 bytes (every plane starts on one)
    CUtensorMap planes;
    const cuuint64_t dims[2] = {MAP_ROW / 2, (cuuint64_t)((size_t)g.count * g.dg_per_leaf / MAP_ROW)};
    const cuuint64_t strides[1] = {MAP_ROW};
    const cuuint32_t box[2] = {MAP_ROW / 2, MAP_BOX}, ones[2] = {1, 1};
    if (g_encode_tiled(&planes, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, ws + g.dg_base, dims, strides, box, ones,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    const int64_t units = leaf_units(g) * g.count;
    int pairs = num_sms / 2;
    if (pairs > ZCTA_MAX / 2) pairs = ZCTA_MAX / 2;  // two product-residue tiles per CTA
    // Whole units to a pair, or (unit, modulus) items and the combine kernel:
    // items as long as every unit's residues fit the product-residue tiles.
    // They fill the pairs evenly, and the combine kernel has the whole GPU
    // where the drain warps of a few pairs end with 50000 clocks of
    // reconstruction.  us a call at 17 moduli, units -> items: leaf of 448 (4
    // units) 172 -> 76, of 1000 (16) 244 -> 125, of 2048 (64) 386 -> 339; 7
    // leaves of 896 (112) 458 -> 394; 3 of 1792 (147, two full rounds of 76
    // pairs) 1063 -> 1051.
    const int split = units <= ZCTA_MAX;
    const size_t smem = (size_t)RNSTAGE * RSTAGE_BYTES + 1024 + 1024;
    const int64_t want = split ? units * LMAX : units;
    if (want < pairs) pairs = (int)want;
    cudaError_t e = launch_chained(crt_gemm_kernel, 2 * pairs, RGEMM_THREADS, smem, stream, tasks_dev, ws, g, planes,
                                   status_dev, split, starve);
    count_launch();
    if (e != cudaSuccess) return e;
    if (split) {
        e = launch_chained(crt_combine_kernel, (unsigned)(units * 2 * 64), 128, 0, stream, tasks_dev, ws, g);
        count_launch();
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

cudaError_t launch_crt_gemm(const LeafTask *tasks_dev, int count, int m, SplitParams p, void *workspace,
                            unsigned int *status_dev, int num_sms, cudaStream_t stream, int starve) {
    const Geo g = make_geo(m, count, p.scheme);
    cudaError_t e = crt_prepare();
    if (e != cudaSuccess) return e;
    // Leaves of one row tile leave a unit's second CTA and half the columns of
    // the first without work, so of a pair's 16 drain warps 4 at most
    // reconstruct.  Many of them go as items, in as few equal launches as the
    // product-residue tiles allow: the combine kernel spreads their
    // reconstruction over the GPU.  us of the GEMM and combine kernels at 17
    // moduli, units -> items (with one-CTA MMAs before both): 16807 leaves of 128
    // 14900 -> 11210 (13600), 2401 of 128 2172 -> 1603 (2000), 2401 of 96 1808 ->
    // 1428 (1780), 16807 of 40 8480 -> 7340 (9580).  Leaves of up to 32
    // reconstruct too little for it: integers of 11 bits, 16807 of 16 2870 ->
    // 3650, of 32 3610 -> 3770, of 40 4080 -> 3870.
    const bool parts = count > ZCTA_MAX && m > 32 && m <= TM;
    const int launches = parts ? (count + ZCTA_MAX - 1) / ZCTA_MAX : 1, per = (count + launches - 1) / launches;
    for (int first = 0; first < count; first += per) {
        Geo part = g;
        part.count = count - first < per ? count - first : per;
        part.sc_base += (size_t)first * g.sc_per_leaf;
        part.dg_base += (size_t)first * g.dg_per_leaf;
        e = launch_crt_gemm_leaves(tasks_dev + first, (char *)workspace, part, status_dev, num_sms, stream, starve);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace caps
