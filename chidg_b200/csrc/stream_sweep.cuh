// ILU programme: streamed task sweeps (CHIDG_SCHED_STREAM).
//
// The work of one triangular sweep is a list of tasks (StreamTask), handed out
// in topological order of the rows they wait for and executed by persistent
// CTAs (several per SM, so that several tasks are in flight on each SM) with a
// producer/consumer split:
//
//   producer (one lane of the last warp)  takes a ticket, and copies the task's
//       blocks column-chunk by column-chunk into a ring of shared-memory stages
//       with cp.async.bulk (completion counted on the stage's mbarrier).  The
//       copy does not depend on the sweep's values, so it runs ahead of the
//       dependency waits: the chunks are in shared memory when the parent row
//       is published.  The next ticket and its descriptor are fetched while
//       the current task's chunks are posted.
//   consumers (the other warps)  wait (bounded) for the parent rows, stage their
//       segments of z, multiply the chunks as they land, release each stage, and
//       at the task's last chunk publish its result.
//
// A sweep is a chain of rows (levels), and where a level holds few rows its
// time is that of one hop: parent published, segment fetched, block
// multiplied, row completed and published.  What is on that path is kept
// short:
//
//   rows of at most SW_ROW_B equations (order 1 with five fields: 40) are one
//       task with all their blocks, inv(D) included in the backward sweep: one
//       flag a row, no partial sums through memory.
//   larger blocks are cut into sweep_slices(b) slices of columns, a task each:
//       135 columns are three slices of 49 KB, 320 columns eight of 102 KB; as
//       one task (146 or 819 KB) most of a block was still to be streamed by
//       one CTA when its parent was published.
//       Where a level has slices enough to fill the chip, a task takes all of a
//       block's slices one after another (the same sums, one wait).
//   a slice leaves its partial sums and counts itself; nobody gathers them on
//       the path: a task that needs the row adds the partials up itself, in
//       order, while it stages them (forward: z_r = v_r - sum of the row's
//       partials; backward: the slices of inv(D_r) stage z_r - sum of the U
//       partials, and the row's children add up the partials of inv(D_r)).
//       The last task of a row to finish writes z_r itself, for whoever reads it
//       later.
//   a task's indices come with its descriptor, not from dependent loads after
//       the wait (an acquire leaves the SM's L1 without them).
//
// The cut depends on the row's own block size and on the kind of preconditioner
// only, so a row sums in the same order whatever matrix or batch it belongs to.
//
// Bound by the copies at 24^3 elements of order 2 (5.8 and 15.8 GB: 1.14 ms
// forward, 2.83 ms backward with matvec rows; with whole blocks as tasks 1.20 and
// 2.85) and by the hops in smaller boxes: 12^3 260 and 491 us (392 and 699), 9 x 8
// x 10 of order 3 346 and 853 us (988 and 2054), 8^3 of order 1 64 and 101 us (103
// and 160).
//
// Deadlock freedom: a task waits only for tasks with smaller tickets.  Each
// CTA consumes its tasks in ticket order, and a producer posts a task's chunks
// as soon as stages free, so the unfinished task with the smallest ticket can
// always proceed.  Every wait (flags, counts, mbarriers) is bounded; on a
// timeout the sweep records status 1 and finishes with wrong values instead of
// hanging.
//
// Bulk copies need 16-byte aligned source, destination and size: each chunk's
// source is rounded down to 16 bytes (the element offset inside the stage is
// carried with the chunk) and its length rounded up; device buffers carry 256
// bytes of slack past their end, so the rounded copies stay inside them.
#pragma once

#include <algorithm>

#include "kernels.cuh"

namespace chidg {

constexpr int SS_MAX_B = 1024;                              // rows per block
constexpr int SS_MAX_STAGES = 8;
constexpr int SS_MAX_NC = 512;                              // consumer threads (16 warps)
constexpr int SS_BLKS = 32;                                 // blocks of a matvec row whose offsets are staged
constexpr int SS_SLOTS = SS_MAX_STAGES + 3;                 // descriptors in flight: a ring of tasks, the one being finished and the next

enum { SW_ENTRY = 0, SW_DIAG = 1, SW_ROW = 2, SW_MATVEC = 3 };   // slice of an entry, of inv(D); whole row; matvec row

constexpr int SW_ROW_B = 64;      // rows of at most this size are one task (SW_ROW) ...
constexpr int SW_ROW_COLS = 384;  // ... if their entries' columns fit the staged segment
// Slices of a block of b rows.  More shorten a hop, but every child of a row adds
// up its partial sums again.  Forward and backward sweep with matvec rows, us: 320
// rows, 8^3, eight 267 / 649, four 289 / 679, three 333 / 738; 9 x 9 x 20, eight 700
// / 1745, four 653 / 1668.  From 161 to 300 rows small boxes and thin ones want
// eight (200 rows, 4^3: eight 59 / 135, five 62 / 150; 162 rows, 60 elements in a
// row: an application 598, with four 697), large boxes fewer (162 rows, 9 x 9 x 20:
// eight 389 / 742, four 291 / 607, whole blocks 380 / 787).
inline int sweep_slices(int b) { return b <= SW_ROW_B ? 1 : b <= 160 ? 3 : 8; }
// RASILU0: many subdomains advance side by side, so its levels are long and its chains
// short; slices of some 80 columns above 160 rows.  Apply, ms, whole blocks / these /
// eight: 12^3 elements in 64 subdomains, 162 rows 0.79 / 0.78 / 0.97, 243 rows 1.57 /
// 1.59 / 1.76, 320 rows 2.68 / 2.72 / 2.88; 8^3 in eight, 320 rows 1.23 / 0.74 / 0.79.
inline int sweep_slices_ras(int b) { return b <= 160 ? sweep_slices(b) : std::min(8, b / 80); }
// Programmes without couplings (Jacobi, precon_HB) have no chain, but the matvec
// rows' wait.  Above 160 rows each of their slices is its own task however many
// there are, which fills the last turn of the CTAs better than whole blocks (1 slice)
// or grouped slices (8g); up to 256 rows eight are too many.  Apply, us, 1 / 3 / 8 /
// 8g: 200 rows, 100 blocks 34 / 31 / 32 / 35, 720 73 / 70 / 85 / 82, 1500 106 / 107 /
// 131 / 119; 320 rows, 100 blocks 55 / 44 / 42 / 43, 720 137 / 120 / 127 / 145, 1500
// 218 / 211 / 222 / 231; 640 rows, 100 blocks 134 / 81 / 80 / 80, 990 559 / 490 / 509
// / 586.  With the matvec rows eight are better than three above 256 rows (320 rows,
// 60 blocks: 40 us a step).  At 135 rows ungrouped slices cost (1500 blocks 70 / 86;
// grouped 75).
inline int sweep_slices_diagonal(int b) { return b > 160 && b <= 256 ? 3 : sweep_slices(b); }
inline bool sweep_groups_slices(int b, bool diagonal) { return !diagonal || b <= 160; }

// A task.  A slice's (or several adjacent slices') staged segment is base[seg + c] -/+ the sum of npart
// partial vectors part[pseg + k * pb + c] (pb: their row's size), c < cols:
// base is z (src 0), v (src 1) or nothing (src 2), the sum subtracted except
// with src 2.  SW_ROW backward: the row's own z comes from z (src 0) or, without
// lower entries, from v (src 1).
struct alignas(16) StreamTask {
    int32_t row, code, b, cols;     // programme row, its size, columns of the slice (SW_ROW forward: of all entries)
    int64_t off;                    // the slice's first value in LD (forward, inv(D)) or A
    int64_t zrow, vrow;             // the row's z and v
    int64_t out, rbase;             // partials this task writes; first partials of its row (for the last task)
    int64_t seg, pseg;
    int32_t par, wait;              // the wait: < 0 none, 0 flag of par, n its count reaching n
    int32_t npart, pb, src, nall;   // nall: tasks of the row (the last one completes it); SW_MATVEC, SW_ROW: U partial vectors of the row at rbase
    int32_t q0, q1;                 // the row's entries
    int32_t nc, s0, nsl, ns;        // slices s0 .. s0 + nsl - 1 of the ns that nc columns are cut into
};

// Device bytes that a row of nlo lower and nup upper entries adds to the sweeps'
// scratch and task lists, at most (the forward, the backward and the list with the
// matvec row)
inline int64_t sweep_row_bytes(int b, int nlo, int nup) {
    const int64_t ns = sweep_slices(b), task = sizeof(StreamTask);
    if (b <= SW_ROW_B) return 8 * (int64_t)b * std::max(nlo, nup) + 4 * task;
    return 8 * b * ns * std::max(nlo, nup + 1) + task * (ns * (nlo + 2 * (nup + 1)) + 2);
}

struct StreamMeta {
    int task;      // descriptor slot, -1 = end of the sweep for this CTA
    int chunk, nchunk;
    int col0, ncols;
    int shift;     // element offset of the chunk inside the stage
    int skip;      // the row's system is frozen: nothing is read, computed or written
    int end;       // last chunk of a slice; SW_ROW backward: last chunk of the U blocks
};

// Rows of frozen systems in a batched solve (a system whose Arnoldi process
// has converged while the others go on): row r belongs to system row_sys[r],
// frozen when active[row_sys[r]] == 0.  The streamed kernels skip such rows:
// no block is copied, no wait is taken, nothing is written, so a step costs
// what its active systems read.  The rows of a system depend only on rows of
// the same system, and a frozen system's vectors are not read again before
// its next restart, so skipping them changes no active system's values.
// Empty (active == nullptr): every row runs.
struct RowMask {
    const int32_t* row_sys = nullptr;
    const int32_t* active = nullptr;
    int nrow = 0;              // rows the map covers
};
__device__ __forceinline__ bool row_frozen(const RowMask& mk, int row) {
    return mk.active != nullptr && mk.active[mk.row_sys[row]] == 0;
}

struct StreamTasks {
    const StreamTask* task;
    unsigned* count;            // per row: completed entry slices
    unsigned* dcount;           // backward: per row, completed slices of inv(D)
};

// the row structure of a matrix whose rows' blocks are stored one after
// another (the streamed matvec's view)
struct MatvecRowsView {
    const int64_t* row_ptr;     // blocks of row i: row_ptr[i] .. row_ptr[i+1]-1
    const int64_t* blk_voff;
    const int64_t* blk_xoff;
    const int32_t* blk_nc;
    const int64_t* row_yoff;
    const int32_t* row_b;
};

// ring of `stages` stages of `stage_bytes` (a multiple of 16), the parent
// segment (xcap values: the largest block of the programme), the row-sum
// scratch (nc values, one per consumer thread), mbarriers and descriptors
__host__ __device__ constexpr size_t stream_xcap(int max_b) { return (size_t)((max_b + 31) / 32) * 32; }
// (max_b: the largest segment staged at once -- a block's columns, or with
// fused matvec rows also a matrix row's columns; a 32-double scratch follows
// the row sums for the fused rows' sums of squares)
__host__ __device__ constexpr size_t stream_smem_bytes(size_t acc_size, int stages, int stage_bytes, int max_b, int nc) {
    return (size_t)stages * stage_bytes + (stream_xcap(max_b) + nc) * acc_size + 32 * sizeof(double) +
           2 * SS_MAX_STAGES * sizeof(uint64_t) + SS_MAX_STAGES * sizeof(StreamMeta) + SS_SLOTS * sizeof(StreamTask) + 64;
}

// columns a chunk of a strip of cols columns (b rows of esz bytes) takes: as
// few chunks as the stage allows, of equal size
__device__ __forceinline__ int chunk_cols(int cols, int b, int esz, int chunk_bytes) {
    const int most = max(1, chunk_bytes / (b * esz));
    const int n = (cols + most - 1) / most;
    return n > 0 ? (cols + n - 1) / n : 1;
}

// The matvec that follows the backward sweep in FGMRES (w = A z_j,
// type_fgmres.f90:175-189), run inside the backward sweep's launch: one task
// per matrix row (SW_MATVEC), handed out after the sweep tasks that publish
// the rows its columns read, so the rows' values stream while the sweep's
// dependency chain waits.
//
// The sweep has already formed the products of row r's upper blocks with z
// (the U partials U_rj z_j, ILU0's U being A's upper blocks,
// precon_ILU0.f90:370-395), and z_j is final when they are formed.  With
// `skip` set (the sweep's U blocks are the matvec's values, same type), the
// matvec row streams only the blocks the sweep did not read -- the diagonal,
// the lower blocks and any others -- and adds the row's U partials, in order,
// to their product: y_r = (A_rr z_r + sum_lower A_rk z_k) + sum_U part.  That
// drops the U blocks' second read (3/7 of the matrix on a hex box).  Chunks
// stay within a block.
template <typename TA, typename TX>
struct FusedMv {
    MatvecRowsView rows;         // the matrix rows (contiguous values per row)
    const TA* val;
    TX* y;
    double* row_sumsq;
    const int32_t* col_prow;     // per block of the matrix: the programme row publishing its column segment
    const uint8_t* skip = nullptr;   // per block of the matrix: 1 = a U block of the sweep, its partial reused
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}
// The waiting thread is suspended (up to the hint, 0.1 ms) until the phase
// completes, so waiting warps do not take issue slots from working ones.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity), "r"(100000u)
        : "memory");
    return ok != 0;
}
// wait until the phase with the given parity has completed; false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, long long limit) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity))
        if (clock64() - t0 > limit) return false;
    return true;
}
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
template <int NC>
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(NC) : "memory"); }
// counter increment that releases the writes ordered before it (this thread's
// and, through the preceding barrier, the other consumers') and acquires the
// writes the other CTAs released with their increments
__device__ __forceinline__ unsigned atom_add_acq_rel(unsigned* p, unsigned v) {
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// the sum over the consumer threads (result in consumer thread 0)
template <int NC>
__device__ __forceinline__ double consumers_sum(double v, double* scratch, int ctid) {
    v = warp_sum(v);
    if ((ctid & 31) == 0) scratch[ctid >> 5] = v;
    consumers_sync<NC>();
    double s = 0.0;
    if (ctid < 32) {
        s = (ctid < NC / 32) ? scratch[ctid] : 0.0;
        s = warp_sum(s);
    }
    return s;
}

// acc[rr] += sum over the chunk's columns of block(r, c) * x(c); rows r of this
// thread as set up by the caller (b <= NC: one row, columns strided by the G
// groups; otherwise rows r + NC*rr, all columns)
template <int NC, int RPT, typename TB, typename ACC>
__device__ __forceinline__ void stream_chunk(const TB* __restrict__ d, const ACC* __restrict__ xs, int b, int ncols, int r,
                                             int g, int G, ACC (&acc)[RPT]) {
    if (b <= NC) {
        if (g >= G) return;
        const TB* col = d + r;
        ACC a0 = acc[0], a1 = 0;
        int c = g;
        for (; c + G < ncols; c += 2 * G) {
            a0 += cvt<ACC>(col[(int64_t)c * b]) * xs[c];
            a1 += cvt<ACC>(col[(int64_t)(c + G) * b]) * xs[c + G];
        }
        if (c < ncols) a0 += cvt<ACC>(col[(int64_t)c * b]) * xs[c];
        acc[0] = a0 + a1;
    } else {
        for (int c = 0; c < ncols; ++c) {
            const ACC x = xs[c];
            #pragma unroll
            for (int rr = 0; rr < RPT; ++rr) {
                const int row = r + NC * rr;
                if (row < b) acc[rr] += cvt<ACC>(d[(int64_t)c * b + row]) * x;
            }
        }
    }
}

// the row sums of this task's product for rows ctid (+ NC*rr), as seen by
// threads ctid < b (b <= NC) or all threads otherwise
template <int NC, int RPT, typename ACC>
__device__ __forceinline__ void stream_reduce(ACC* red, int b, int r, int g, int G, int ctid, ACC (&acc)[RPT]) {
    if (b <= NC) {
        if (g < G) red[g * b + r] = acc[0];
        consumers_sync<NC>();
        if (ctid < b) {
            ACC s = 0;
            for (int gg = 0; gg < G; ++gg) s += red[gg * b + ctid];
            acc[0] = s;
        }
    }
}

// s + n partial vectors (stride b) in order; eight loads go out together
template <typename ACC>
__device__ __forceinline__ ACC sum_partials_at(const ACC* p, int n, int b, ACC s) {
    constexpr int U = 8;
    for (int k0 = 0; k0 < n; k0 += U) {
        ACC v[U];
        #pragma unroll
        for (int k = 0; k < U; ++k) v[k] = k0 + k < n ? ld_cg(p + (int64_t)(k0 + k) * b) : ACC(0);
        #pragma unroll
        for (int k = 0; k < U; ++k)
            if (k0 + k < n) s += v[k];
    }
    return s;
}
// wait (one thread) until *p has reached target; false on timeout
__device__ __forceinline__ bool wait_count(const unsigned* p, unsigned target, long long limit) {
    if ((int)(ld_acquire(p) - target) >= 0) return true;
    const long long t0 = clock64();
    for (int k = 0; (int)(ld_acquire(p) - target) < 0; ++k) {
        if (clock64() - t0 > limit) return false;
        if (k > 16) __nanosleep(32);
    }
    return true;
}
__device__ __forceinline__ void red_release(unsigned* p, unsigned n) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(n) : "memory");
}

// CW consumer warps; `stages` stages of `stage_bytes` bytes each.  MV: the
// backward sweep also runs the matvec rows of F (tasks SW_MATVEC).
template <typename TL, typename TU, typename TX, typename ACC, bool FORWARD, int CW, typename TA = double, bool MV = false>
__global__ void __launch_bounds__(32 * CW + 32, CW == 16 ? 2 : CW == 8 ? 4 : 7)   // CTAs an SM: what the rings leave room for
    k_ilu_stream(IluRows R, const TL* __restrict__ LD, const TU* __restrict__ Aval, StreamTasks T, int ntasks,
                 const TX* __restrict__ v, TX* __restrict__ zx, ACC* __restrict__ part, SweepSync S, int nstage,
                 int stage_bytes, int max_b, FusedMv<TA, TX> F, RowMask mask) {
    constexpr int NC = 32 * CW;                  // consumer threads
    static_assert(NC <= SS_MAX_NC, "row-sum scratch");
    static_assert(!(MV && FORWARD), "matvec rows run in the backward sweep");
    constexpr int RPT = (SS_MAX_B + NC - 1) / NC;
    extern __shared__ __align__(128) unsigned char ss_smem[];
    unsigned char* stages = ss_smem;
    StreamTask* slots = reinterpret_cast<StreamTask*>(ss_smem + (size_t)nstage * stage_bytes);
    double* scratch = reinterpret_cast<double*>(slots + SS_SLOTS);   // 32 doubles
    uint64_t* full = reinterpret_cast<uint64_t*>(scratch + 32);
    uint64_t* empty = full + SS_MAX_STAGES;
    ACC* xs = reinterpret_cast<ACC*>(empty + SS_MAX_STAGES);
    ACC* red = xs + stream_xcap(max_b);          // G*b <= NC row sums
    StreamMeta* meta = reinterpret_cast<StreamMeta*>(red + NC);
    __shared__ int s_last;
    __shared__ int s_nc[SS_BLKS];                // SW_MATVEC: columns and x offsets (-1: not staged) of the row's blocks
    __shared__ int64_t s_x[SS_BLKS];
    const int chunk_bytes = stage_bytes - 16;    // payload before rounding out to 16 bytes

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < nstage; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, CW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == CW) {
        // ------------------------------------------------------------ producer
        if (lane != 0) return;
        int stage = 0, slot = 0;
        unsigned phase = 0;
        unsigned t = atomicAdd(S.counter, 1u);
        // descriptors live in shared memory; the next one's slot is free: the ring
        // and the consumers hold fewer tasks than there are slots
        if (t < (unsigned)ntasks) slots[0] = T.task[t];
        while (t < (unsigned)ntasks) {
            const StreamTask& d = slots[slot];
            unsigned tn = 0;
            const int b = d.b;
            int ch = 0, nchunk = 0;
            // columns [col0, col0 + ncols) of the staged segment times the strip at src
            auto post = [&](const void* from, int col0, int ncols, int esz, int end, int skip) {
                // the next ticket, its latency under the wait for the last
                // chunk's stage: not earlier, or a long task would keep a
                // short one waiting that another CTA could take
                if (ch == nchunk - 1) tn = atomicAdd(S.counter, 1u);
                if (!mbar_wait(empty + stage, phase ^ 1u, S.spin_limit)) atomicExch(S.status, 1);
                StreamMeta m;
                m.task = slot; m.chunk = ch; m.nchunk = nchunk;
                m.col0 = col0; m.ncols = ncols; m.skip = skip; m.end = end;
                const uintptr_t src = reinterpret_cast<uintptr_t>(from);
                const uintptr_t a0 = src & ~(uintptr_t)15;
                m.shift = ncols > 0 ? (int)(src - a0) / esz : 0;
                meta[stage] = m;
                if (ncols > 0) {
                    const unsigned bytes = (unsigned)((size_t)ncols * b * esz);
                    const unsigned len = (unsigned)(((src - a0) + bytes + 15) & ~(uintptr_t)15);
                    mbar_arrive_expect_tx(full + stage, len);
                    bulk_copy_g2s(stages + (size_t)stage * stage_bytes, reinterpret_cast<const void*>(a0), len, full + stage);
                } else {
                    mbar_arrive(full + stage);
                }
                ++ch;
                if (++stage == nstage) { stage = 0; phase ^= 1u; }
            };
            // a strip of cols columns, staged from column col0 on; its last chunk carries `end`
            auto post_strip = [&](const void* base, int col0, int cols, int esz, int end) {
                const int kc = chunk_cols(cols, b, esz, chunk_bytes);
                for (int c = 0; c < cols; c += kc)
                    post(reinterpret_cast<const unsigned char*>(base) + (size_t)c * b * esz, col0 + c, min(kc, cols - c), esz,
                         c + kc >= cols ? end : 0, 0);
            };
            auto chunks = [&](int cols, int esz) {
                const int kc = chunk_cols(cols, b, esz, chunk_bytes);
                return (cols + kc - 1) / kc;
            };
            if (row_frozen(mask, d.row)) {
                // a frozen system's row: one empty chunk, nothing read or written
                nchunk = 1;
                post(nullptr, 0, 0, 1, 0, 1);
            } else if (MV && d.code == SW_MATVEC) {
                // the row's blocks, with F.skip only those the sweep did not read
                const int64_t k0 = F.rows.row_ptr[d.row], k1 = F.rows.row_ptr[d.row + 1];
                for (int64_t k = k0; k < k1; ++k)
                    if (F.skip == nullptr || !F.skip[k]) nchunk += chunks(F.rows.blk_nc[k], sizeof(TA));
                int col = 0;
                for (int64_t k = k0; k < k1; ++k) {
                    const int nc = F.rows.blk_nc[k];
                    if (F.skip == nullptr || !F.skip[k]) post_strip(F.val + F.rows.blk_voff[k], col, nc, sizeof(TA), 0);
                    col += nc;
                }
                if (nchunk == 0) { nchunk = 1; post(nullptr, 0, 0, 1, 0, 0); }   // nothing streamed
            } else if (d.code == SW_ROW) {
                if (FORWARD) {
                    // the row's L blocks follow one another in LD
                    nchunk = max(1, chunks(d.cols, sizeof(TL)));
                    if (d.cols == 0) post(nullptr, 0, 0, 1, 0, 0);
                    else post_strip(LD + d.off, 0, d.cols, sizeof(TL), 0);
                } else {
                    for (int e = d.q0; e < d.q1; ++e) nchunk += chunks(R.up_nc[e], sizeof(TU));
                    nchunk += chunks(b, sizeof(TL));
                    int col = 0;
                    for (int e = d.q0; e < d.q1; ++e) {
                        post_strip(Aval + R.up_U[e], col, R.up_nc[e], sizeof(TU), e == d.q1 - 1);
                        col += R.up_nc[e];
                    }
                    post_strip(LD + d.off, 0, b, sizeof(TL), 0);
                }
            } else {
                const int esz = (FORWARD || d.code == SW_DIAG) ? (int)sizeof(TL) : (int)sizeof(TU);
                // slices s0 .. s0 + nsl - 1 of the cut of nc columns, side by side
                const int ns = d.ns;
                auto cut = [&](int s) { return d.nc * (d.s0 + s) / ns - d.nc * d.s0 / ns; };
                for (int s = 0; s < d.nsl; ++s) nchunk += max(1, chunks(cut(s + 1) - cut(s), esz));
                for (int s = 0; s < d.nsl; ++s) {
                    const int c0 = cut(s), cols = cut(s + 1) - c0;
                    const int64_t o = d.off + (int64_t)c0 * b;
                    if (cols == 0) post(nullptr, 0, 0, 1, 1, 0);
                    else if (FORWARD || d.code == SW_DIAG) post_strip(LD + o, c0, cols, esz, 1);
                    else post_strip(Aval + o, c0, cols, esz, 1);
                }
            }
            if (++slot == SS_SLOTS) slot = 0;
            t = tn;
            if (t < (unsigned)ntasks) slots[slot] = T.task[t];
        }
        if (!mbar_wait(empty + stage, phase ^ 1u, S.spin_limit)) atomicExch(S.status, 1);
        meta[stage].task = -1;
        mbar_arrive(full + stage);
        return;
    }

    // ---------------------------------------------------------------- consumers
    const int ctid = tid;
    int stage = 0;
    unsigned phase = 0;
    int slot = 0, b = 0, G = 1, r = 0, g = 0;
    int sl = 0;                                  // slice of the task being summed; SW_ROW: 1 once U is done
    TX own = TX(0);                              // SW_ROW: the row's v (forward) or z (backward), fetched before the wait
    ACC acc[RPT];
    for (;;) {
        if (!mbar_wait(full + stage, phase, S.spin_limit)) { if (ctid == 0) atomicExch(S.status, 1); }
        const StreamMeta m = meta[stage];
        if (m.task < 0) break;
        if (m.skip) {
            // a frozen system's row: release the stage, nothing else
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + stage);
            if (++stage == nstage) { stage = 0; phase ^= 1u; }
            continue;
        }
        slot = m.task;
        const StreamTask& d = slots[slot];
        const int code = d.code;
        if (m.chunk == 0) {
            b = d.b;
            sl = 0;
            if (b <= NC) { G = NC / b; r = ctid % b; g = ctid / b; }
            else { G = 1; r = ctid; g = 0; }
            #pragma unroll
            for (int rr = 0; rr < RPT; ++rr) acc[rr] = 0;
            if (MV && code == SW_MATVEC) {
                // every column segment of the row published by the sweep, then staged
                // (the blocks' offsets fetched before the wait)
                const int64_t k0 = F.rows.row_ptr[d.row], k1 = F.rows.row_ptr[d.row + 1];
                const int nb = (int)(k1 - k0);
                if (nb <= SS_BLKS) {
                    if (ctid < nb) {
                        s_nc[ctid] = F.rows.blk_nc[k0 + ctid];
                        s_x[ctid] = (F.skip == nullptr || !F.skip[k0 + ctid]) ? F.rows.blk_xoff[k0 + ctid] : -1;
                    }
                    if (ctid < nb && !wait_flag(S.flags, F.col_prow[k0 + ctid], S.epoch, S.spin_limit)) atomicExch(S.status, 1);
                    consumers_sync<NC>();
                    // the segments side by side; four loads of a thread go out together
                    int total = 0;
                    for (int k = 0; k < nb; ++k) total += s_nc[k];
                    for (int c0 = ctid; c0 < total; c0 += 4 * NC) {
                        TX val4[4];
                        #pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            int c = c0 + u * NC, k = 0;
                            while (k < nb && c >= s_nc[k]) c -= s_nc[k++];
                            val4[u] = (k < nb && s_x[k] >= 0) ? ld_cg(zx + s_x[k] + c) : TX(0);
                        }
                        #pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (c0 + u * NC < total) xs[c0 + u * NC] = cvt<ACC>(val4[u]);
                    }
                } else {
                    for (int64_t k = k0 + ctid; k < k1; k += NC)
                        if (!wait_flag(S.flags, F.col_prow[k], S.epoch, S.spin_limit)) atomicExch(S.status, 1);
                    consumers_sync<NC>();
                    int off = 0;
                    for (int64_t k = k0; k < k1; ++k) {
                        const int nc = F.rows.blk_nc[k];
                        if (F.skip == nullptr || !F.skip[k]) {
                            const TX* xp = zx + F.rows.blk_xoff[k];
                            for (int c = ctid; c < nc; c += NC) xs[off + c] = cvt<ACC>(ld_cg(xp + c));
                        }
                        off += nc;
                    }
                }
            } else if (code == SW_ROW) {
                // thread c stages column c of the entries' columns side by side
                // (and c + NC): its address before the wait
                const int32_t* par = FORWARD ? R.lo_par : R.up_par;
                const int32_t* ncs = FORWARD ? R.lo_nc : R.up_nc;
                constexpr int CPT = (SW_ROW_COLS + NC - 1) / NC;
                const TX* at[CPT];
                #pragma unroll
                for (int u = 0; u < CPT; ++u) at[u] = nullptr;
                int off = 0;
                for (int e = d.q0; e < d.q1; ++e) {
                    const int nc = ncs[e];
                    const TX* zp = zx + R.z_off[par[e]];
                    #pragma unroll
                    for (int u = 0; u < CPT; ++u) {
                        const int c = ctid + u * NC - off;
                        if (c >= 0 && c < nc) at[u] = zp + c;
                    }
                    off += nc;
                }
                if (ctid < b) own = (FORWARD || d.src == 1) ? v[d.vrow + ctid] : zx[d.zrow + ctid];
                for (int e = d.q0 + ctid; e < d.q1; e += NC)
                    if (!wait_flag(S.flags, par[e], S.epoch, S.spin_limit)) atomicExch(S.status, 1);
                consumers_sync<NC>();
                #pragma unroll
                for (int u = 0; u < CPT; ++u)
                    if (at[u] != nullptr) xs[ctid + u * NC] = cvt<ACC>(ld_cg(at[u]));
                if (!FORWARD && d.q1 == d.q0 && ctid < b) xs[ctid] = cvt<ACC>(own);      // inv(D) alone
            } else {
                // slice of an entry or of inv(D): see StreamTask
                const int wt = d.wait;
                if (ctid == 0 && wt >= 0) {
                    const unsigned* p = (FORWARD ? T.count : code == SW_DIAG ? T.count : T.dcount) + d.par;
                    if (!(wt == 0 ? wait_flag(S.flags, d.par, S.epoch, S.spin_limit) : wait_count(p, (unsigned)wt, S.spin_limit)))
                        atomicExch(S.status, 1);
                }
                consumers_sync<NC>();
                const TX* base = (d.src == 1 ? v : zx) + d.seg;
                const ACC* pp = part + d.pseg;
                for (int c = ctid; c < d.cols; c += NC) {
                    const double x0 = d.src == 2 ? 0.0 : to_d(ld_cg(base + c));
                    const ACC s = sum_partials_at(pp + c, d.npart, d.pb, ACC(0));
                    xs[c] = cvt<ACC>(from_d<TX>(d.src == 2 ? (double)s : x0 - (double)s));
                }
            }
            consumers_sync<NC>();
        }
        if (!FORWARD && code == SW_ROW && sl == 1) {
            // the row's U products are complete: t_r = z_r - sum takes the segments' place
            stream_reduce<NC, RPT>(red, b, r, g, G, ctid, acc);
            if (ctid < b) {
                part[d.out + ctid] = acc[0];                // read by the row's matvec task
                xs[ctid] = cvt<ACC>(from_d<TX>(to_d(own) - (double)acc[0]));
            }
            acc[0] = 0;
            sl = 2;
            consumers_sync<NC>();
        }
        if (m.ncols > 0) {
            const unsigned char* sb = stages + (size_t)stage * stage_bytes;
            if (MV && code == SW_MATVEC)
                stream_chunk<NC, RPT, TA, ACC>(reinterpret_cast<const TA*>(sb) + m.shift, xs + m.col0, b, m.ncols, r, g, G, acc);
            else if (FORWARD || code == SW_DIAG || (code == SW_ROW && (sl == 2 || d.q1 == d.q0)))
                stream_chunk<NC, RPT, TL, ACC>(reinterpret_cast<const TL*>(sb) + m.shift, xs + m.col0, b, m.ncols, r, g, G, acc);
            else
                stream_chunk<NC, RPT, TU, ACC>(reinterpret_cast<const TU*>(sb) + m.shift, xs + m.col0, b, m.ncols, r, g, G, acc);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + stage);
        if (++stage == nstage) { stage = 0; phase ^= 1u; }
        if (m.chunk != m.nchunk - 1) {
            if (!m.end) continue;
            if (code == SW_ROW) { sl = 1; continue; }
            // a slice with others after it in the task: its partial sums
            stream_reduce<NC, RPT>(red, b, r, g, G, ctid, acc);
            ACC* o = part + d.out + (int64_t)sl * b;
            #pragma unroll
            for (int rr = 0; rr < RPT; ++rr) {
                const int i = (b <= NC) ? (rr == 0 ? ctid : b) : ctid + NC * rr;
                if (i < b) o[i] = acc[rr];
                acc[rr] = 0;
            }
            ++sl;
            consumers_sync<NC>();        // the row sums' scratch is written again
            continue;
        }

        // ------------------------------------------------ the task's last chunk
        stream_reduce<NC, RPT>(red, b, r, g, G, ctid, acc);
        if (MV && code == SW_MATVEC) {
            // y_r = A_r z and its sum of squares (with F.skip: plus the row's U partials, in order)
            double sq = 0.0;
            const int64_t yo = F.rows.row_yoff[d.row];
            #pragma unroll
            for (int rr = 0; rr < RPT; ++rr) {
                const int i = (b <= NC) ? (rr == 0 ? ctid : b) : ctid + NC * rr;
                if (i < b) {
                    if (F.skip != nullptr) acc[rr] += sum_partials_at(part + d.rbase + i, d.nall, b, ACC(0));
                    const TX o = from_d<TX>((double)acc[rr]);
                    F.y[yo + i] = o;
                    const double od = to_d(o);
                    sq += od * od;
                }
            }
            if (F.row_sumsq != nullptr) {
                const double s2 = consumers_sum<NC>(sq, scratch, ctid);
                if (ctid == 0) F.row_sumsq[d.row] = s2;
            }
            consumers_sync<NC>();        // xs, red and scratch are reused by the next task
            continue;
        }
        if (code == SW_ROW) {
            // the row is complete: z_r = v_r - sum, or inv(D_r) t_r
            if (ctid < b) {
                const double x = FORWARD ? to_d(own) - (double)acc[0] : (double)acc[0];
                zx[d.zrow + ctid] = from_d<TX>(x);
            }
            consumers_sync<NC>();
            if (ctid == 0) st_release(S.flags + d.row, S.epoch);
            continue;
        }
        // the slice's partial sums, counted; the last forward slice, or slice of
        // inv(D), of the row writes z_r
        const bool none = FORWARD && d.q1 == d.q0;         // a row without entries: z_r = v_r
        if (none) {}
        else {
            ACC* o = part + d.out + (int64_t)sl * b;
            if (b <= NC) { if (ctid < b) o[ctid] = acc[0]; }
            else {
                #pragma unroll
                for (int rr = 0; rr < RPT; ++rr)
                    if (ctid + NC * rr < b) o[ctid + NC * rr] = acc[rr];
            }
        }
        consumers_sync<NC>();
        if (!FORWARD && code == SW_ENTRY) {
            if (ctid == 0) red_release(T.count + d.row, (unsigned)d.nsl);
            continue;
        }
        if (ctid == 0)
            s_last = atom_add_acq_rel((FORWARD ? T.count : T.dcount) + d.row, (unsigned)d.nsl) + (unsigned)d.nsl == (unsigned)d.nall;
        consumers_sync<NC>();
        if (!s_last) continue;
        for (int i = ctid; i < b; i += NC) {
            const ACC s = sum_partials_at(part + d.rbase + i, none ? 0 : d.nall, b, ACC(0));
            zx[d.zrow + i] = from_d<TX>(FORWARD ? to_d(v[d.vrow + i]) - (double)s : (double)s);
        }
        consumers_sync<NC>();
        if (ctid == 0) st_release(S.flags + d.row, S.epoch);
    }
}

}  // namespace chidg
