// The whole FP64 factorisation of a programme of small blocks (at most FR_MAX
// rows: order 1 with five fields) in one launch.
//
// Level by level such a factorisation is three launches a wavefront whose
// kernels last 10 to 30 us, a small box's wavefronts far from filling the
// chip.  Here persistent CTAs take the rows in factorisation order; a row waits
// (bounded) for the inverses of its lower parents, forms its L blocks, its D
// and D's inverse with the code of the level-by-level kernels (fg_tile, gj_block:
// the same sums in the same order, so a block's factors do not depend on which
// of the two forms computed them) and publishes itself.  A row waits only for
// rows with smaller tickets, whose holders are running: no deadlock.
//
// Bound by a row's chain of latencies times the wavefronts (40 rows: 48 us a
// row, 26 of them the inverse) until the boxes fill the chip.  Factorisation,
// level by level and here, in ms: 40-row blocks 2^3 elements 0.19, 0.13; 10 x 9
// x 8 1.38, 1.07; 18^3 3.24, 2.35; 24^3 4.80, 3.53; 8 rows 18^3 1.61, 0.70; 54
// rows 14^3 3.02, 2.62; 64 rows 14^3 3.25, 2.97, 24^3 7.36, 5.99.  Larger blocks
// keep the three launches: their products are several CTA tiles and their
// inverse wants more warps than the tile has.  With profiling on the launch counts
// as factorisation only: its products and inverses are not launches of their own.
#pragma once

#include "factor_gemm.cuh"
#include "inverse_gj.cuh"

#include <algorithm>

namespace chidg {

constexpr int FR_MAX = 64;
constexpr int FR_T = 2;                                       // panel warps of the inverse, as launch_inverse gives them

inline size_t fr_smem(int b) { return std::max(FG_SMEM, gj_smem(b, 1)); }

struct FactorRows {
    const GemmTask *ltasks, *stasks;      // in row order; stasks one a row
    const GemmPair *lpairs, *spairs;
    const int32_t* rows;                  // factorisation order
    const int32_t *prow_b, *prow_elem, *lo_ptr, *lo_par, *ltask_of;   // ltask_of: first L task of the row at a position
    const int64_t* dinv_off;
    int nrows;
};

static __global__ void __launch_bounds__(FG_THREADS)
    k_factor_rows(FactorRows R, const double* Aval, double* LD, SweepSync S, int* __restrict__ status) {
    extern __shared__ __align__(128) unsigned char fr_raw[];
    __shared__ int s_pos;
    double* fg = reinterpret_cast<double*>(fr_raw);
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_pos = (int)atomicAdd(S.counter, 1u);
        __syncthreads();
        const int pos = s_pos;
        if (pos >= R.nrows) break;
        const int pr = R.rows[pos], b = R.prow_b[pr], q0 = R.lo_ptr[pr], nl = R.lo_ptr[pr + 1] - q0, l0 = R.ltask_of[pos];
        for (int q = tid; q < nl; q += FG_THREADS)
            if (!wait_flag(S.flags, R.lo_par[q0 + q], S.epoch, S.spin_limit)) atomicExch(S.status, 1);
        __syncthreads();
        for (int q = 0; q < nl; ++q) {
            fg_tile(R.ltasks[l0 + q], 0, 0, pos, R.lpairs, Aval, LD, nullptr, LD, 1.0, fg);
            __syncthreads();
        }
        fg_tile(R.stasks[pos], 0, 0, pos, R.spairs, LD, Aval, Aval, LD, -1.0, fg);
        __syncthreads();
        gj_block<false, 4>(fr_raw, LD + R.dinv_off[pr], b, R.prow_elem[pr], status, 1, FR_T);
        // the barriers' memory is used again: by the next row's tiles
        __syncthreads();
        if (tid == 0) {
            GjShared& sh = *reinterpret_cast<GjShared*>(fr_raw);
            for (uint64_t* m = sh.ready; m != sh.la + 2; ++m)
                asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(m)) : "memory");
            __threadfence();
            st_release(S.flags + pr, S.epoch);
        }
        __syncthreads();
    }
}

}  // namespace chidg
