// Plain form base case: C = A * B on FP64 DMMA tensor cores (mma.sync f64).
//
// Replaces block_multiply -> square_dgemm_zero -> dgemm_ (multiply.cpp:
// 1082-1141, dgemm-blas.cpp:4-13): column-major m x m operands, beta = 0;
// and the rectangular subproject's base case localRectMM (rect-class/
// rectmm.cpp:47-51): A m x k, B k x n, C m x n, column-major, beta = 0.
//
// GB300 runs FP64 (DFMA and DMMA alike) at ~1.1 TFLOP/s for the whole GPU,
// about 1.8 multiply-adds per clock per SM, so this kernel is bound by the
// DMMA pipe at any sensible tiling; a 16-deep K slab in shared memory (the
// next one already in registers) keeps operand traffic far below what that
// pipe can consume.  What a launch loses is therefore work for padding and
// SMs with one tile more than the others.  8 x 8 blocks of C outside the leaf
// and 4-deep steps beyond K are skipped (a 14 x 14 leaf in a 64 x 64 tile took
// 29 us, 49 of them 97 % of an n = 56 multiply), and the default tile is
// chosen per launch (pick_tile).  A CTA is a WM x WN grid of warps, each FM x
// FN blocks of m8n8k4, one CTA per tile of one leaf of the batch (blockIdx.z).
// Every tile accumulates each entry over k in the same order, so they agree
// bit for bit.  The epilogue applies the task's fold (DmmaFold) of the lean
// 'd' step that consumes the product.
#include "common.cuh"

namespace caps {

namespace {
constexpr int BK = 16;

__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
    asm volatile(
        "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}
}  // namespace

template <int WM, int WN, int FM, int FN>
__global__ void __launch_bounds__(32 * WM * WN) dmma_gemm_kernel(const DmmaTask *__restrict__ tasks, int m, int n,
                                                                 int k) {
    constexpr int BM = 8 * FM * WM, BN = 8 * FN * WN, NT = 32 * WM * WN;
    constexpr int PA = BM * BK / NT, PB = BN * BK / NT;  // operand entries a thread loads per slab
    constexpr int LDA = BM + 8, LDB = BN + 8;  // padded rows (banks)
    __shared__ double As[BK][LDA];  // As[k][i]
    __shared__ double Bs[BK][LDB];  // Bs[k][j]
    chain_wait();
    const DmmaTask t = tasks[blockIdx.z];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = warp / WN, wc = warp % WN;
    const int64_t i0 = (int64_t)blockIdx.y * BM, j0 = (int64_t)blockIdx.x * BN;
    const int64_t M = m, N = n, K = k;  // A: M x K, B: K x N, C: M x N
    // this warp's 8 x 8 blocks inside the leaf
    const int64_t rows = M - i0 - 8 * FM * wr, cols = N - j0 - 8 * FN * wc;
    const int fm = rows >= 8 * FM ? FM : rows > 0 ? (int)(rows + 7) / 8 : 0;
    const int fn = cols >= 8 * FN ? FN : cols > 0 ? (int)(cols + 7) / 8 : 0;
    const bool whole = fm == FM && fn == FN;

    double acc[FM][FN][2];
#pragma unroll
    for (int a = 0; a < FM; a++)
#pragma unroll
        for (int b = 0; b < FN; b++) acc[a][b][0] = acc[a][b][1] = 0.0;

    double pa[PA], pb[PB];  // the next slab
    auto fetch = [&](int64_t k0) {
        // A tile: BM rows x 16 k from a column-major source; consecutive
        // threads read consecutive rows of one column
#pragma unroll
        for (int p = 0; p < PA; p++) {
            const int e = tid + NT * p, row = e % BM, kk = e / BM;
            const int64_t gi = i0 + row, gk = k0 + kk;
            pa[p] = (gi < M && gk < K) ? t.A[gi + gk * M] : 0.0;
        }
        // B tile: 16 k x BN columns; consecutive threads read the 16 k of one column
#pragma unroll
        for (int p = 0; p < PB; p++) {
            const int e = tid + NT * p, kk = e % BK, col = e / BK;
            const int64_t gk = k0 + kk, gj = j0 + col;
            pb[p] = (gk < K && gj < N) ? t.B[gk + gj * K] : 0.0;
        }
    };
    fetch(0);
    for (int64_t k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int p = 0; p < PA; p++) As[(tid + NT * p) / BM][(tid + NT * p) % BM] = pa[p];
#pragma unroll
        for (int p = 0; p < PB; p++) Bs[(tid + NT * p) % BK][(tid + NT * p) / BK] = pb[p];
        __syncthreads();
        if (k0 + BK < K) fetch(k0 + BK);
        if (whole && k0 + BK <= K) {
#pragma unroll
            for (int ks = 0; ks < BK; ks += 4) {
                double af[FM], bf[FN];
#pragma unroll
                for (int a = 0; a < FM; a++) af[a] = As[ks + (lane & 3)][8 * FM * wr + 8 * a + (lane >> 2)];
#pragma unroll
                for (int b = 0; b < FN; b++) bf[b] = Bs[ks + (lane & 3)][8 * FN * wc + 8 * b + (lane >> 2)];
#pragma unroll
                for (int a = 0; a < FM; a++)
#pragma unroll
                    for (int b = 0; b < FN; b++) dmma_8x8x4(acc[a][b], af[a], bf[b]);
            }
        } else {
            const int kend = K - k0 < BK ? (int)(K - k0) : BK;
#pragma unroll 1
            for (int ks = 0; ks < kend; ks += 4) {
                double bf[FN];
#pragma unroll
                for (int b = 0; b < FN; b++) bf[b] = Bs[ks + (lane & 3)][8 * FN * wc + 8 * b + (lane >> 2)];
#pragma unroll
                for (int a = 0; a < FM; a++) {
                    if (a >= fm) break;  // warp-uniform, as below
                    const double af = As[ks + (lane & 3)][8 * FM * wr + 8 * a + (lane >> 2)];
#pragma unroll
                    for (int b = 0; b < FN; b++)
                        if (b < fn) dmma_8x8x4(acc[a][b], af, bf[b]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < FM; a++)
#pragma unroll
        for (int b = 0; b < FN; b++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int64_t gi = i0 + 8 * FM * wr + 8 * a + (lane >> 2);
                const int64_t gj = j0 + 8 * FN * wc + 8 * b + 2 * (lane & 3) + e;
                if (gi >= M || gj >= N) continue;
                const int64_t x = gi + gj * M;
                const double p = acc[a][b][e];
                switch (t.fold) {
                    case FOLD_ADD: t.C[x] = t.s0[x] + p; break;
                    case FOLD_SUB: t.C[x] = t.s0[x] - p; break;
                    case FOLD_ADD2: {
                        const double u2 = t.s0[x], u1 = t.s1[x];
                        t.C[x] = u2 + p;
                        t.d1[x] = u1 + p;
                        break;
                    }
                    default: t.C[x] = p;
                }
            }
}

template <int WM, int WN, int FM, int FN>
static cudaError_t launch_dmma_shape(const DmmaTask *tasks_dev, int count, int m, int n, int k, cudaStream_t stream) {
    constexpr int BM = 8 * FM * WM, BN = 8 * FN * WN;
    const unsigned rows = (unsigned)((m + BM - 1) / BM), cols = (unsigned)((n + BN - 1) / BN);
    for (int base = 0; base < count; base += 65535) {
        const int c = count - base < 65535 ? count - base : 65535;
        dim3 grid(cols, rows, (unsigned)c);
        launch_chained(dmma_gemm_kernel<WM, WN, FM, FN>, grid, 32 * WM * WN, 0, stream, tasks_dev + base, m, n, k);
        count_launch();
    }
    return cudaGetLastError();
}

// The square tile side whose busiest SM has the least to do.  The CTAs of an
// SM share its one DMMA pipe, so a launch takes as long as the SM with the
// most tile area: a leaf of 1024 is 256 tiles of 64 on 152 SMs, 2 on the
// busiest and 1.7 on average; of 32, 1024 tiles, 7 and 6.7.  Smaller tiles read their
// operands more often and synchronise more per multiply-add, which costs next
// to nothing at this pipe's rate (4096 x 2048 x 3072: 46890 us with 16, 47010
// with 32).  us a multiply, 64 always -> picked: n = 4096 'dd' (leaves of 1024)
// 121390 -> 96920 (32 alone: 97100; 93100 at the pipe's rate), leaf of 1500 7040
// -> 6270, 4096 x 2048 x 3072 48910 -> 46890, n = 56 'dd' 1471 -> 437 (with the
// skipped padding).
//
// Row tiles go in grid.y, which holds 65535 of them: a tall, narrow product
// (the rectangular base case; 1048561 x 8 is 65536 row tiles of 16) takes the
// best side whose row tiles fit.
static int pick_tile(int count, int m, int n) {
    const int64_t max_rows = 65535;
    const int sides[3] = {64, 32, 16};
    const double cost[3] = {1.0, 1.01, 1.005};
    int best = 64;
    double best_t = 0.0;
    for (int i = 0; i < 3; i++) {
        const int64_t t = sides[i], rows = (m + t - 1) / t;
        if (i > 0 && rows > max_rows) continue;
        const int64_t ctas = rows * ((n + t - 1) / t) * (int64_t)count;
        const double busiest = (double)((ctas + 151) / 152) * (double)(t * t) * cost[i];
        if (i == 0 || busiest < best_t) {
            best = sides[i];
            best_t = busiest;
        }
    }
    return best;
}

// a tuned tile's shape; 64 x 64, the largest it takes, for the pick per launch
void dmma_tile_shape(int tile, int *rows, int *cols) {
    switch (tile) {
        case DMMA_TILE_32x32: *rows = 32; *cols = 32; break;
        case DMMA_TILE_128x64: *rows = 128; *cols = 64; break;
        default: *rows = 64; *cols = 64; break;
    }
}

cudaError_t launch_dmma_rect(const DmmaTask *tasks_dev, int count, int m, int n, int k, cudaStream_t stream,
                             int tile) {
    if (count <= 0 || m <= 0 || n <= 0) return cudaSuccess;
    switch (tile) {
        case DMMA_TILE_32x32: return launch_dmma_shape<2, 2, 2, 2>(tasks_dev, count, m, n, k, stream);
        case DMMA_TILE_128x64: return launch_dmma_shape<4, 2, 4, 4>(tasks_dev, count, m, n, k, stream);
        case DMMA_TILE_64x64: return launch_dmma_shape<2, 2, 4, 4>(tasks_dev, count, m, n, k, stream);
    }
    switch (pick_tile(count, m, n)) {
        case 16: return launch_dmma_shape<2, 2, 1, 1>(tasks_dev, count, m, n, k, stream);
        case 32: return launch_dmma_shape<2, 2, 2, 2>(tasks_dev, count, m, n, k, stream);
        default: return launch_dmma_shape<2, 2, 4, 4>(tasks_dev, count, m, n, k, stream);
    }
}

cudaError_t launch_dmma_gemm(const DmmaTask *tasks_dev, int count, int m, cudaStream_t stream, int tile) {
    return launch_dmma_rect(tasks_dev, count, m, m, m, stream, tile);
}

}  // namespace caps
