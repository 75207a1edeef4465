// In-place inverses of the diagonal blocks (mod_inv.f90:97-150), up to
// GJ_MAX rows: Gauss-Jordan with partial (row) pivoting in panels of eight
// columns, one block per cluster of C CTAs (one CTA where the block fits its
// shared memory).
//
// A CTA keeps its share of the block's columns (whole 8-column tiles) in
// shared memory, column-major.  Its first T warps (a row of the block per
// thread) eliminate the panels it owns, the other warps apply finished panels
// to its columns:
//
//   panel J   the rows are in registers, eight columns a thread.  A step's
//             pivot is the entry of largest magnitude among the rows not yet
//             used as pivots (the first such row on ties): the pivot DGETRF
//             selects.  Every lane takes the reciprocal of its own entry
//             while the warp looks for its best row, the winner's row and
//             reciprocal go to a buffer of the step's parity, and one barrier
//             of the T warps later every warp picks the winner among them.
//             The columns rotate by one a step, so the loop over the eight
//             steps stays compact (unrolled, its instruction fetches cost
//             more than its arithmetic).  Rows are not interchanged; step k
//             records its row p_k.
//   update    every other column c changes by the panel's eight steps as
//             a_c <- a_c with rows {p_k} zeroed + P X_c, P the eliminated
//             panel and X_c the old values of a_c in rows p_k: m8n8k4 FP64
//             tensor-core products, a warp a tile of eight columns.
//
// Look-ahead: the panel warps apply panel J to tile J + 1 themselves (each
// thread its own row, the panel's row still in registers) and go on, while the
// update warps apply it to the others, tile J + 2 first.  The
// critical path is the chain of panels (eight barriers each); the products
// (2 b^3 operations) run beside it.  Panels are double-buffered and handed
// over by mbarriers; in a cluster the owner's panel is pushed into the other
// CTAs' buffers by bulk copies between shared memories, counted on their
// mbarriers.
//
// Bound by that chain (654 cycles a pivot step at 40 rows, 1035 at 135: the
// latencies of a barrier, a reduction over the warp and eight dependent
// multiply-adds), not by the FP64 rate or by memory; the pivots' divisions run
// beside the warps' search and cost nothing measurable against a seed and a
// correction step (28.0, 96.4 and 279 us a launch of 40, 135 and 320 rows; 28.8,
// 97.2 and 283).  A launch of up to 148 blocks takes 28 us at 40 rows (54 with one
// step per barrier pair over the whole block), 96 us at 135 rows (142), 279 us at
// 320 rows for as many blocks as clusters of five fit the chip (24 to 29).  Levels
// of many more blocks above 208 rows are inverted by inverse_rows.cuh, one CTA a
// block.  All levels of 9 x 8 x 10 elements of order 3 take 12.0 ms, 31.4 in that
// form alone.
//
// After the last panel the stored matrix S satisfies S(p_k, j) =
// inv(A)(k, p_j); the write-back undoes the permutation.  A zero pivot records
// the element in *status (ESINGULAR) and leaves garbage; a NaN entry is taken
// as pivot so the NaN propagates.  Every mbarrier wait is bounded; one that
// runs out is reported the same way, and the waits after it give up at once.
#pragma once

#include "kernels.cuh"
#include "stream_sweep.cuh"

namespace chidg {

constexpr int GJ_MAX = 384;                       // rows: 12 panel warps
constexpr int GJ_MAXT = GJ_MAX / 32;
constexpr int GJ_THREADS = 512;                   // at most
constexpr long long GJ_WAIT_LIMIT = 1ll << 31;    // clock cycles

__host__ __device__ __forceinline__ int gj_rows(int b) { return (b + 15) / 16 * 16; }   // padded rows
// doubles of a panel buffer: eight columns of stride gj_rows + 4 and the eight pivot rows (ints)
__host__ __device__ __forceinline__ int gj_panel(int b) { return 8 * (gj_rows(b) + 4) + 8; }

struct alignas(16) GjShared {
    uint64_t ready[2], freed[2], la[2];           // panel landed; panel buffer read by all; tile ready for look-ahead
    // per step parity and panel warp: the candidate's row, its reciprocal and
    // (low word of the value, row index) as the words of a double
    double crow[2][GJ_MAXT][10];
    alignas(16) unsigned chi[2][GJ_MAXT];         // its key: high word of the value (0: no candidate)
    int pivrow[GJ_MAX];                           // step -> row
    alignas(16) double X[8][8];                   // the next tile's values in the panel's pivot rows
};

inline size_t gj_smem(int b, int C) {
    const int tiles = ((b + 7) / 8 + C - 1) / C;
    return sizeof(double) * ((size_t)tiles * 8 * (gj_rows(b) + 2) + 2 * (size_t)gj_panel(b)) + sizeof(GjShared);
}
// the smallest cluster whose CTAs hold a block of b rows
inline int gj_cluster(int b) {
    for (int C = 1; C <= 8; ++C)
        if (gj_smem(b, C) <= 227 * 1024) return C;
    return 0;
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <bool CL>
__device__ __forceinline__ void gj_arrive(uint64_t* bar, uint32_t rank) {
    if (CL)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr(bar, rank)) : "memory");
    else
        mbar_arrive(bar);
}
// bounded wait for a phase; limit drops to 0 once a wait has run out
template <bool CL>
__device__ __forceinline__ void gj_wait(uint64_t* bar, unsigned parity, long long& limit) {
    if (!CL) {
        if (!mbar_wait(bar, parity, limit)) limit = 0;
        return;
    }
    const long long t0 = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_addr(bar)), "r"(parity), "r"(100000u)
            : "memory");
        if (ok) return;
        if (clock64() - t0 > limit) { limit = 0; return; }
    }
}

// two doubles to shared memory where p is set, without a branch
__device__ __forceinline__ void gj_store2(bool p, double* at, double x, double y) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.shared.v2.f64 [%1], {%2, %3};\n\t}" ::"r"((int)p),
                 "r"(smem_addr(at)), "d"(x), "d"(y)
                 : "memory");
}

// a pivot row of a panel's header (-1: no step), also if the panel never came
__device__ __forceinline__ int gj_pivot(int p, int b) { return (unsigned)p < (unsigned)b ? p : -1; }
// parity of the phase of panel J's barriers (per parity of J, one phase for
// every panel from the third on that the CTA owns)
__device__ __forceinline__ unsigned gj_phase(int J, int first) {
    const int jl = max(first, 2);
    return (unsigned)((J - (jl + ((jl ^ J) & 1))) >> 1) & 1u;
}

// operands of rows r16 .. r16 + 15 of an 8-column tile (stride LD) and of the panel P (stride LDP)
__device__ __forceinline__ void gj_mma_rows(const double* S, int LD, const double* P, int LDP, int r16, int g, int tq,
                                            double (&d)[4], double (&a)[4]) {
    const double* s = S + 2 * tq * LD + r16 + g;
    d[0] = s[0];
    d[1] = s[LD];
    d[2] = s[8];
    d[3] = s[LD + 8];
    const double* p = P + tq * LDP + r16 + g;
    a[0] = p[0];
    a[1] = p[8];
    a[2] = p[4 * LDP];
    a[3] = p[4 * LDP + 8];
}

// one block D (b x b, column-major) in place, by the CTAs of a cluster of C
// (CL) or one CTA; T of the CTA's warps are the panel warps (MAXT: at least T, a
// multiple of 4).  raw: gj_smem(b, C) bytes.
template <bool CL, int MAXT>
__device__ __forceinline__ void gj_block(unsigned char* gj_raw, double* D, int b, int elem, int* status, int C, int T) {
    GjShared& sh = *reinterpret_cast<GjShared*>(gj_raw);
    const uint32_t rank = CL ? cluster_rank() : 0;
    const int nt8 = (b + 7) / 8, tc = (nt8 + C - 1) / C;          // tiles of the block, of a CTA
    const int first = min((int)rank * tc, nt8), ntl = min(tc, nt8 - first);
    const int rp = gj_rows(b), LD = rp + 2, LDP = rp + 4, PB = gj_panel(b);
    double* P0 = reinterpret_cast<double*>(gj_raw + sizeof(GjShared));   // two panel buffers
    double* S = P0 + 2 * PB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5, NU = nw - T - (CL ? 1 : 0);
    const int g = lane >> 2, tq = lane & 3;
    long long limit = GJ_WAIT_LIMIT;
    bool singular = false;

    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(sh.ready + s, 1);
            mbar_init(sh.freed + s, nw * C);
            mbar_init(sh.la + s, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < GJ_MAX; i += blockDim.x) sh.pivrow[i] = i;   // an index even if a wait gives up
    if (tid < 2 * GJ_MAXT) sh.chi[tid / GJ_MAXT][tid % GJ_MAXT] = 0u;   // warps that are not there propose nothing
    // the CTA's columns, zero in the padding
    for (int c = warp; c < 8 * ntl; c += nw) {
        const int col = 8 * first + c;
        for (int i = lane; i < rp; i += 32) cp_async8(S + c * LD + i, D + i + (int64_t)col * b, i < b && col < b);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if (CL) cluster_barrier();

    if (warp < T) {
        // ------------------------------------------------------------ panels
        const int i = tid;
        const bool mine = i < b;
        bool used = false;
        auto panel_sync = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(32 * T) : "memory"); };
        double r[8], sn[8];                       // the row in tile J, in tile J + 1
        // r <- the row of a tile (sn, 0 if it was the pivot of step `step` of the
        // panel before) + the panel's row pv times the tile's pivot rows in sh.X
        auto apply_panel = [&](const double (&pv)[8], int step) {
            double t[8];
            #pragma unroll
            for (int c = 0; c < 8; ++c) t[c] = step >= 0 ? 0.0 : sn[c];
            #pragma unroll
            for (int k = 0; k < 8; ++k) {
                #pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double2 x = reinterpret_cast<const double2*>(sh.X[k])[c];
                    t[2 * c] = fma(pv[k], x.x, t[2 * c]);
                    t[2 * c + 1] = fma(pv[k], x.y, t[2 * c + 1]);
                }
            }
            #pragma unroll
            for (int c = 0; c < 8; ++c) r[c] = t[c];
        };
        auto give_x = [&](int step) {
            if (step < 0) return;
            #pragma unroll
            for (int c = 0; c < 4; ++c) reinterpret_cast<double2*>(sh.X[step])[c] = make_double2(sn[2 * c], sn[2 * c + 1]);
        };
        bool have = false;                        // r is tile J with the panel before it applied
        for (int J = 0; J < nt8; ++J) {
            const bool own = J >= first && J < first + ntl;
            double* St = S + (J - first) * 8 * LD;
            if (J > 0 && !have) {
                // a panel of another CTA
                const double* P = P0 + ((J - 1) & 1) * PB;
                const int* hdr = reinterpret_cast<const int*>(P + 8 * LDP);
                gj_wait<CL>(sh.ready + ((J - 1) & 1), (unsigned)((J - 1) >> 1) & 1u, limit);
                int step = -1;
                #pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (hdr[k] == i) step = k;
                used = used || step >= 0;
                if (own) {
                    if (J >= 2) gj_wait<CL>(sh.la + (J & 1), gj_phase(J, first), limit);
                    double pv[8];
                    #pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        sn[c] = i < rp ? St[c * LD + i] : 0.0;
                        pv[c] = i < rp ? P[c * LDP + i] : 0.0;
                    }
                    give_x(step);
                    panel_sync();
                    apply_panel(pv, step);
                }
                __syncwarp();
            }
            if (J > 0 && lane == 0 && J + 1 < nt8) gj_arrive<CL>(sh.freed + ((J - 1) & 1), (J + 1) / tc);
            if (!own) continue;
            if (J == 0) {
                #pragma unroll
                for (int c = 0; c < 8; ++c) r[c] = i < rp ? St[c * LD + i] : 0.0;
            }
            const bool next = J + 1 < first + ntl;
            int mystep = -1;
            #pragma unroll 1
            for (int kk = 0; kk < 8; ++kk) {
                if (kk == 5) {
                    // the next tile's row, and the panel buffer, both long ready as a rule
                    if (next) {
                        if (J + 1 >= 2) gj_wait<CL>(sh.la + ((J + 1) & 1), gj_phase(J + 1, first), limit);
                        #pragma unroll
                        for (int c = 0; c < 8; ++c) sn[c] = i < rp ? St[(8 + c) * LD + i] : 0.0;
                    }
                    if (J >= 2) gj_wait<CL>(sh.freed + (J & 1), gj_phase(J, first), limit);
                }
                if (8 * J + kk >= b) {
                    // past the last column: only the rotation
                    const double t = r[0];
                    #pragma unroll
                    for (int c = 0; c < 7; ++c) r[c] = r[c + 1];
                    r[7] = t;
                    continue;
                }
                const int buf = kk & 1;
                // keys: the bits of |v| are monotone in |v| (a NaN sorts above
                // infinity); the top bit marks a candidate.  The lanes holding
                // the largest high word write at once; only if there are several
                // (checked beside that) do the low words decide
                const unsigned hi = (mine && !used) ? (unsigned)__double2hiint(r[0]) | 0x80000000u : 0u;
                const unsigned lo = (unsigned)__double2loint(r[0]);
                // (opaque, or the compiler divides by a padding row's zero after all: the
                // division's slow path, 5 to 10 % of a step)
                double div = hi != 0u ? r[0] : 1.0;
                asm("" : "+d"(div));
                const double rcp = 1.0 / div;
                const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
                const bool top = hi == mhi && hi != 0u;
                auto propose = [&](bool mine_) {
                    double* cr = sh.crow[buf][warp];
                    #pragma unroll
                    for (int c = 0; c < 4; ++c) gj_store2(mine_, cr + 2 * c, r[2 * c], r[2 * c + 1]);
                    gj_store2(mine_, cr + 8, rcp, __hiloint2double((int)lo, i));
                };
                propose(top);
                if (lane == 0) sh.chi[buf][warp] = mhi;
                const unsigned tops = __ballot_sync(0xffffffffu, top);
                if (tops & (tops - 1)) {
                    const unsigned mlo = __reduce_max_sync(0xffffffffu, top ? lo : 0u);
                    const unsigned best = __ballot_sync(0xffffffffu, top && lo == mlo);
                    __syncwarp();
                    propose(lane == __ffs(best) - 1);
                }
                panel_sync();
                // the warps' keys, by a tree (the first warp on ties); equal high
                // words are looked for beside it
                unsigned key[MAXT];
                int idx[MAXT];
                #pragma unroll
                for (int q = 0; q < MAXT; q += 4) {
                    const uint4 k4 = reinterpret_cast<const uint4*>(sh.chi[buf])[q / 4];
                    key[q] = k4.x; key[q + 1] = k4.y; key[q + 2] = k4.z; key[q + 3] = k4.w;
                }
                const unsigned mykey = sh.chi[buf][lane < MAXT ? lane : 0];
                #pragma unroll
                for (int q = 0; q < MAXT; ++q) idx[q] = q;
                #pragma unroll
                for (int n = MAXT; n > 1; n = (n + 1) / 2)
                    #pragma unroll
                    for (int q = 0; q < n / 2; ++q) {
                        const bool up = key[2 * q + 1] > key[2 * q];
                        key[q] = up ? key[2 * q + 1] : key[2 * q];
                        idx[q] = up ? idx[2 * q + 1] : idx[2 * q];
                        if (2 * q + 3 == n) { key[q + 1] = key[2 * q + 2]; idx[q + 1] = idx[2 * q + 2]; }
                    }
                const unsigned gh = key[0];
                int ww = idx[0];
                double pr[8], rc;
                int p;
                auto take = [&]() {
                    const double2* cr = reinterpret_cast<const double2*>(sh.crow[buf][ww]);
                    #pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const double2 v = cr[c];
                        pr[2 * c] = v.x;
                        pr[2 * c + 1] = v.y;
                    }
                    const double2 v = cr[4];
                    rc = v.x;
                    p = __double2loint(v.y);
                };
                take();
                const unsigned eq = __ballot_sync(0xffffffffu, lane < MAXT && mykey == gh);
                if (eq & (eq - 1)) {
                    auto low = [&](int q) { return (unsigned)__double2hiint(sh.crow[buf][q][9]); };
                    unsigned gl = low(ww);
                    for (int q = ww + 1; q < T; ++q)
                        if (sh.chi[buf][q] == gh && low(q) > gl) { gl = low(q); ww = q; }
                    take();
                }
                if (pr[0] == 0.0) { singular = true; rc = 1.0; }
                // the pivot row becomes its scaled self, the others lose their multiple of it
                const bool is_p = i == p;
                const double m = is_p ? -rc : r[0] * rc;
                #pragma unroll
                for (int c = 0; c < 7; ++c) r[c] = fma(-m, pr[c + 1], is_p ? 0.0 : r[c + 1]);
                r[7] = -m;
                if (is_p) { used = true; mystep = kk; }
            }
            double* P = P0 + (J & 1) * PB;
            int* hdr = reinterpret_cast<int*>(P + 8 * LDP);
            if (i < rp) {
                #pragma unroll
                for (int c = 0; c < 8; ++c) {
                    St[c * LD + i] = r[c];
                    P[c * LDP + i] = r[c];
                }
            }
            if (mystep >= 0) hdr[mystep] = i;
            if (i < 8 && 8 * J + i >= b) hdr[i] = -1;
            if (next) give_x(mystep);
            if (CL) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            panel_sync();
            if (tid == 0) mbar_arrive(sh.ready + (J & 1));
            if (next) {
                double pv[8];
                #pragma unroll
                for (int c = 0; c < 8; ++c) pv[c] = r[c];
                apply_panel(pv, mystep);
            }
            have = next;
        }
    } else if (CL && warp == nw - 1) {
        // ------------------------------------------------------------ this CTA's panels to the others
        // (a warp of its own: as part of a panel warp's work the pushes took as
        // long as five pivot steps a panel).  It follows every panel and counts as
        // a reader of each, so that it never falls a phase behind
        for (int J = 0; J < nt8; ++J) {
            gj_wait<CL>(sh.ready + (J & 1), (unsigned)(J >> 1) & 1u, limit);
            if (J >= first && J < first + ntl && lane < C && lane != (int)rank && limit != 0) {
                const double* P = P0 + (J & 1) * PB;
                const uint32_t bytes = (uint32_t)(PB * sizeof(double)), bar = cluster_addr(sh.ready + (J & 1), lane);
                asm volatile("mbarrier.arrive.expect_tx.release.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                             : "memory");
                asm volatile(
                    "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        cluster_addr(P, lane)),
                    "r"(smem_addr(P)), "r"(bytes), "r"(bar)
                    : "memory");
            }
            __syncwarp();
            if (lane == 0 && J + 2 < nt8) gj_arrive<CL>(sh.freed + (J & 1), (J + 2) / tc);
        }
    } else {
        // ------------------------------------------------------------ updates
        const int u = warp - T;
        for (int J = 0; J < nt8; ++J) {
            gj_wait<CL>(sh.ready + (J & 1), (unsigned)(J >> 1) & 1u, limit);
            const double* P = P0 + (J & 1) * PB;
            const int* hdr = reinterpret_cast<const int*>(P + 8 * LDP);
            if (u == 0 && lane < 8 && gj_pivot(hdr[lane], b) >= 0) sh.pivrow[8 * J + lane] = hdr[lane];
            const int pa = gj_pivot(hdr[tq], b), pb = gj_pivot(hdr[tq + 4], b);
            const int start = (J + 2 >= first && J + 2 < first + ntl) ? J + 2 - first : 0;
            for (int tt = 0; tt < ntl; ++tt) {
                const int t = start + tt < ntl ? start + tt : start + tt - ntl, gt = first + t;
                if (t % NU != u || gt == J || gt == J + 1) continue;
                double* St = S + t * 8 * LD;
                const double b0 = pa >= 0 ? St[g * LD + pa] : 0.0, b1 = pb >= 0 ? St[g * LD + pb] : 0.0;
                __syncwarp();
                if (pa >= 0) St[g * LD + pa] = 0.0;
                if (pb >= 0) St[g * LD + pb] = 0.0;
                __syncwarp();
                #pragma unroll 3
                for (int r16 = 0; r16 < rp; r16 += 16) {
                    double d[4], a[4];
                    gj_mma_rows(St, LD, P, LDP, r16, g, tq, d, a);
                    dmma_8x8x4(d[0], d[1], a[0], b0);
                    dmma_8x8x4(d[2], d[3], a[1], b0);
                    dmma_8x8x4(d[0], d[1], a[2], b1);
                    dmma_8x8x4(d[2], d[3], a[3], b1);
                    double* s = St + 2 * tq * LD + r16 + g;
                    s[0] = d[0];
                    s[LD] = d[1];
                    s[8] = d[2];
                    s[LD + 8] = d[3];
                }
                __syncwarp();
                if (gt == J + 2 && lane == 0) mbar_arrive(sh.la + (gt & 1));
            }
            __syncwarp();
            if (lane == 0 && J + 2 < nt8) gj_arrive<CL>(sh.freed + (J & 1), (J + 2) / tc);
        }
    }
    if (limit == 0) singular = true;
    if (singular && lane == 0) atomicMin(status, elem);
    __syncthreads();
    if (CL) cluster_barrier();                    // no CTA leaves while another may write to its shared memory
    // inv(A)(k, p_j) = S(p_k, j); the lane's pivots are the same in every column
    int pk[GJ_MAXT];
    #pragma unroll
    for (int q = 0; q < GJ_MAXT; ++q) pk[q] = lane + 32 * q < b ? sh.pivrow[lane + 32 * q] : 0;
    for (int c = warp; c < 8 * ntl; c += nw) {
        const int col = 8 * first + c;
        if (col >= b) break;
        double* out = D + (int64_t)sh.pivrow[col] * b + lane;
        #pragma unroll
        for (int q = 0; q < GJ_MAXT; ++q)
            if (lane + 32 * q < b) out[32 * q] = S[c * LD + pk[q]];
    }
}

template <bool CL, int MAXT>
static __global__ void __launch_bounds__(GJ_THREADS, 1)
    k_block_inverse_gj(double* __restrict__ LD_, const int64_t* __restrict__ dinv_off, const int32_t* __restrict__ prow_b,
                       const int32_t* __restrict__ prow_elem, const int32_t* __restrict__ rows, int row_begin,
                       int* __restrict__ status, int C, int T) {
    extern __shared__ __align__(128) unsigned char gj_raw[];
    const int prow = rows[row_begin + (CL ? blockIdx.x / C : blockIdx.x)];
    gj_block<CL, MAXT>(gj_raw, LD_ + dinv_off[prow], prow_b[prow], prow_elem[prow], status, C, T);
}

}  // namespace chidg
