// FP64 factor products (precon_ILU0.f90:111-265) on the FP64 tensor cores, for
// every block size: C(m x n) = [Cinit] + sgn * sum_q A_q(m x k_q) B_q(k_q x n)
// over a task list (GemmTask / GemmPair), all operands column-major blocks.
//
// A task's output is cut into tiles of at most 80 x 80 (counted in 8 x 8
// accumulator tiles and balanced: 135 rows are 64 + 71, 320 rows four times
// 80), one CTA of four warps a tile, a warp a quarter of it (at most 40 x 40).
// What bounds it is the FP64 pipe: a slice of K = 8 of a full warp tile takes
// 800 cycles of the warp's sub-core against 20 fragment loads.  The operands are staged 16 columns of K at a
// time by 8-byte cp.async (blocks of odd row counts have column strides that
// are not a multiple of 16 bytes), three stages; three CTAs share an SM, so
// one CTA's staging, first loads and stores run under another's MMAs -- with
// one CTA of 136 x 136 an SM spent more than half of its time between them.
// The smaller tiles also spread a short wavefront over the chip: a 135-row
// product is four CTAs, a 320-row one sixteen.
//
// Shared-memory strides: A is [k][m] with stride 84 and B [n][k] with stride
// 20 doubles, both 4 mod 16, so that the 4 x 4 addresses of a half-warp's
// fragment load fall in 16 distinct banks.
//
// Measured against the kernels it replaced (one CTA of 136 x 136 up to 136
// rows; a SIMT kernel of 64 x 64 tiles above), products of one factorisation:
// 24^3 box of order 2 (391 GFLOP) 22.4 against 34.8 ms (17.5 TFLOP/s), 13 x 14
// x 12 of order 2 4.7 against 8.8 ms, 9 x 8 x 10 of order 3 (252 GFLOP) 10.4
// against 21.7 ms (24 TFLOP/s), 8^3 of order 1 0.61 against 0.95 ms.  A
// wavefront of 320-row products keeps the FP64 pipe busy 77 % of the time, one
// of 135-row products 55 %: short K (nine chunks) and the tail of the last
// CTAs are what is left there.
#pragma once

#include "kernels.cuh"

namespace chidg {

constexpr int FG_T = 10;                       // 8 x 8 accumulator tiles per side of a CTA tile
constexpr int FG_M = 8 * FG_T;
constexpr int FG_W = FG_T / 2;                 // per side of a warp's quarter
constexpr int FG_KC = 16, FG_STAGES = 3, FG_THREADS = 128;
constexpr int FG_LDA = FG_M + 4, FG_LDB = FG_KC + 4;
constexpr int FG_STAGE = FG_KC * FG_LDA + FG_M * FG_LDB;     // doubles
constexpr size_t FG_SMEM = sizeof(double) * FG_STAGES * FG_STAGE;
static_assert(FG_STAGES * FG_STAGE >= FG_M * FG_LDA, "the output tile takes the stages' place");

// CTA tiles along a side of len rows
__host__ __device__ __forceinline__ int fg_parts(int len) { return ((len + 7) / 8 + FG_T - 1) / FG_T; }

// one CTA's tile of one task, as its warps see it
struct FgTile {
    GemmTask t;
    int r0, c0, m, n;          // rows [r0, r0 + m), columns [c0, c0 + n) of the output
    int wi0, wj0;              // the warp's first 8 x 8 tile
};

// chunk (K from k0 of a pair) into a stage.  Rows past m and columns past n
// are not staged (they only reach accumulators that are not stored); k past
// the operands' K is staged as zeros (a copy of no bytes reads nothing).
__device__ __forceinline__ void fg_issue(const FgTile& T, const GemmPair& pr, int k0, const double* Abase,
                                         const double* Bbase, double* as, int lane, int warp) {
    double* bs = as + FG_KC * FG_LDA;
    const int kc = pr.k - k0;
    const double* A = Abase + pr.a_off + T.r0 + (int64_t)(k0 + warp) * T.t.m + lane;
    as += warp * FG_LDA + lane;
    const int64_t astep = 4 * (int64_t)T.t.m;
    #pragma unroll
    for (int u = 0; u < FG_KC / 4; ++u, A += astep) {
        const bool in = warp + 4 * u < kc;
        #pragma unroll
        for (int r = 0; r < 3; ++r)
            if (lane + 32 * r < T.m) cp_async8(as + 4 * u * FG_LDA + 32 * r, A + 32 * r, in);
    }
    const int bk = lane & 15, bj = 2 * warp + (lane >> 4);      // lanes walk K, a half-warp a column
    const double* B = Bbase + pr.b_off + k0 + bk + (int64_t)(T.c0 + bj) * pr.k;
    bs += bj * FG_LDB + bk;
    const int64_t bstep = 8 * (int64_t)pr.k;
    #pragma unroll
    for (int u = 0; u < FG_M / 8; ++u, B += bstep)
        if (bj + 8 * u < T.n) cp_async8(bs + 8 * u * FG_LDB, B, bk < kc);
}

// acc(TI x TJ tiles) += A B over one slice of K = 8: row tiles in pairs by
// m16n8k8, an odd one by two m8n8k4
template <int TI, int TJ>
__device__ __forceinline__ void fg_slice(double (&acc)[TI][TJ][2], const double* a, const double* b) {
    double a0[TI], a1[TI], b0[TJ], b1[TJ];
    #pragma unroll
    for (int i = 0; i < TI; ++i) { a0[i] = a[8 * i]; a1[i] = a[4 * FG_LDA + 8 * i]; }
    #pragma unroll
    for (int j = 0; j < TJ; ++j) { b0[j] = b[8 * j * FG_LDB]; b1[j] = b[4 + 8 * j * FG_LDB]; }
    #pragma unroll
    for (int i = 0; i + 1 < TI; i += 2)
        #pragma unroll
        for (int j = 0; j < TJ; ++j)
            dmma_16x8x8(acc[i][j][0], acc[i][j][1], acc[i + 1][j][0], acc[i + 1][j][1], a0[i], a0[i + 1], a1[i], a1[i + 1],
                        b0[j], b1[j]);
    if (TI & 1) {
        constexpr int i = TI - 1;
        #pragma unroll
        for (int j = 0; j < TJ; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a0[i], b0[j]);
        #pragma unroll
        for (int j = 0; j < TJ; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a1[i], b1[j]);
    }
}

// The walk over K of a warp holding TI x TJ tiles (none: it only stages), its
// sums left in the CTA's output tile in shared memory (column-major, stride
// FG_LDA, over the stages).  K is one list of chunks over all pairs; chunk
// c + 2 is on its way while chunk c feeds the tensor cores (the first two
// turns only stage).  Every warp of the CTA takes the same number of chunks,
// hence the same barriers.  The CTA's warps run up to four of these
// instantiations side by side (a quarter has 5 or 4 tiles a side for 135
// rows), so their code is kept short: an instance that also held the stores
// to memory made the 135-row products wait on instruction fetches.
template <int TI, int TJ>
__device__ __forceinline__ void fg_walk(const FgTile& T, const GemmPair* __restrict__ pairs, int nchunk, const double* Abase,
                                        const double* Bbase, double* smem) {
    constexpr bool WORK = TI > 0 && TJ > 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    double acc[WORK ? TI : 1][WORK ? TJ : 1][2];
    if constexpr (WORK) {
        #pragma unroll
        for (int i = 0; i < TI; ++i)
            #pragma unroll
            for (int j = 0; j < TJ; ++j) { acc[i][j][0] = 0.0; acc[i][j][1] = 0.0; }
    }
    int lq = T.t.q_begin, lk0 = 0, cq = lq, ck0 = 0;      // next chunk to stage, to multiply
    int fill = 0, stage = 0;
    #pragma unroll 1
    for (int c = 1 - FG_STAGES; c < nchunk; ++c) {
        cp_async_wait<FG_STAGES - 2>();
        __syncthreads();                          // chunk c has landed, and every warp is done with chunk c - 1
        if (c + FG_STAGES - 1 < nchunk) {
            const GemmPair pr = pairs[lq];
            fg_issue(T, pr, lk0, Abase, Bbase, smem + fill * FG_STAGE, lane, warp);
            lk0 += FG_KC;
            if (lk0 >= pr.k) { lk0 = 0; ++lq; }
            fill = fill + 1 == FG_STAGES ? 0 : fill + 1;
        }
        cp_async_commit();
        if (c < 0) continue;
        const int k = pairs[cq].k;
        if constexpr (WORK) {
            const double* a = smem + stage * FG_STAGE + tq * FG_LDA + 8 * T.wi0 + g;
            const double* b = smem + stage * FG_STAGE + FG_KC * FG_LDA + (8 * T.wj0 + g) * FG_LDB + tq;
            fg_slice<TI, TJ>(acc, a, b);
            if (k - ck0 > 8) fg_slice<TI, TJ>(acc, a + 8 * FG_LDA, b + 8);
        }
        ck0 += FG_KC;
        if (ck0 >= k) { ck0 = 0; ++cq; }
        stage = stage + 1 == FG_STAGES ? 0 : stage + 1;
    }
    __syncthreads();                              // the stages become the output tile
    if constexpr (WORK) {
        double* o = smem + (8 * T.wj0 + 2 * tq) * FG_LDA + 8 * T.wi0 + g;
        #pragma unroll
        for (int j = 0; j < TJ; ++j)
            #pragma unroll
            for (int i = 0; i < TI; ++i) {
                o[8 * j * FG_LDA + 8 * i] = acc[i][j][0];
                o[(8 * j + 1) * FG_LDA + 8 * i] = acc[i][j][1];
            }
    }
}

// CTA tile (im, in) of task t, by the FG_THREADS threads of a CTA; rot turns the
// warps' quarters.  smem: FG_STAGES * FG_STAGE doubles.
__device__ __forceinline__ void fg_tile(const GemmTask& t, int im, int in, int rot, const GemmPair* __restrict__ pairs,
                                        const double* Abase, const double* Bbase, const double* Cinit, double* Cbase,
                                        double sgn, double* fg_smem) {
    FgTile T;
    T.t = t;
    // the CTA's 8 x 8 tiles [ti0, ti0 + tm) x [tj0, tj0 + tn) of the output
    const int pm = fg_parts(T.t.m), pn = fg_parts(T.t.n);
    if (im >= pm || in >= pn) return;
    const int t8m = (T.t.m + 7) / 8, t8n = (T.t.n + 7) / 8;
    const int ti0 = t8m * im / pm, tj0 = t8n * in / pn;
    const int tm = t8m * (im + 1) / pm - ti0, tn = t8n * (in + 1) / pn - tj0;
    T.r0 = 8 * ti0;
    T.c0 = 8 * tj0;
    T.m = min(8 * tm, T.t.m - T.r0);
    T.n = min(8 * tn, T.t.n - T.c0);
    // the warp's quarter; the larger quarters of odd tile counts rotate over
    // the warps (the sub-cores) with the CTA
    const int role = ((threadIdx.x >> 5) + rot) & 3;
    const int hm = (tm + 1) / 2, hn = (tn + 1) / 2;
    T.wi0 = (role & 1) ? hm : 0;
    T.wj0 = (role >> 1) ? hn : 0;
    const int ti = (role & 1) ? tm - hm : hm, tj = (role >> 1) ? tn - hn : hn;
    int nchunk = 0;
    for (int q = T.t.q_begin; q < T.t.q_end; ++q) nchunk += (pairs[q].k + FG_KC - 1) / FG_KC;
    const double* Ci = T.t.cinit_off >= 0 ? Cinit + T.t.cinit_off + T.r0 + (int64_t)T.c0 * T.t.m : nullptr;
    if (Ci != nullptr)                            // read at the end: into L2 meanwhile
        for (int i = threadIdx.x; i < T.n * 8; i += FG_THREADS) {
            const int r = (i & 7) * 16;
            if (r < T.m) asm volatile("prefetch.global.L2 [%0];" ::"l"(Ci + r + (int64_t)(i >> 3) * T.t.m));
        }
    switch (ti * 8 + tj) {
#define CHIDG_FG(I, J) case I * 8 + J: fg_walk<I, J>(T, pairs, nchunk, Abase, Bbase, fg_smem); break;
#define CHIDG_FG_ROW(I) CHIDG_FG(I, 1) CHIDG_FG(I, 2) CHIDG_FG(I, 3) CHIDG_FG(I, 4) CHIDG_FG(I, 5)
        CHIDG_FG_ROW(1) CHIDG_FG_ROW(2) CHIDG_FG_ROW(3) CHIDG_FG_ROW(4) CHIDG_FG_ROW(5)
#undef CHIDG_FG_ROW
#undef CHIDG_FG
        default: fg_walk<0, 0>(T, pairs, nchunk, Abase, Bbase, fg_smem);
    }
    __syncthreads();
    // a warp a column, consecutive lanes on consecutive rows
    const int lane = threadIdx.x & 31;
    double* C = Cbase + T.t.c_off + T.r0 + (int64_t)T.c0 * T.t.m;
    for (int j0 = threadIdx.x >> 5; j0 < T.n; j0 += 16) {
        double ci[4][3];
        #pragma unroll
        for (int u = 0; u < 4; ++u)
            #pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int j = j0 + 4 * u, i = lane + 32 * r;
                ci[u][r] = (Ci != nullptr && j < T.n && i < T.m) ? Ci[i + (int64_t)j * T.t.m] : 0.0;
            }
        #pragma unroll
        for (int u = 0; u < 4; ++u)
            #pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int j = j0 + 4 * u, i = lane + 32 * r;
                if (j < T.n && i < T.m) C[i + (int64_t)j * T.t.m] = ci[u][r] + sgn * fg_smem[j * FG_LDA + i];
            }
    }
}

static __global__ void __launch_bounds__(FG_THREADS, 3)
    k_task_gemm_f64(const GemmTask* __restrict__ tasks, const GemmPair* __restrict__ pairs, int parts_m, int parts_n,
                    const double* Abase, const double* Bbase, const double* Cinit, double* Cbase, double sgn) {
    extern __shared__ __align__(16) double fg_smem[];
    const int tiles = parts_m * parts_n, tile = blockIdx.x % tiles;
    fg_tile(tasks[blockIdx.x / tiles], tile % parts_m, tile / parts_m, blockIdx.x, pairs, Abase, Bbase, Cinit, Cbase, sgn,
            fg_smem);
}

}  // namespace chidg
