// chidg_gpu.cu -- host side of the B200-native ChiDG linear-solve path:
// C ABI objects (context, chidg_matrix, chidg_vector, preconditioners) and the
// programme builders that turn the reference's block-ILU0 / RAS+ILU0 loops into
// level-scheduled GPU sweeps.  The FGMRES driver lives in fgmres.cu.
#include "chidg_gpu_internal.cuh"
#include "inverse_rows.cuh"

#include <tuple>
#include <type_traits>

#include <atomic>

#include <algorithm>
#include <chrono>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <unordered_map>

using namespace chidg;

// ---------------------------------------------------------------------------
// context
// ---------------------------------------------------------------------------
int chidg::fail(chidg_gpu_ctx* ctx, int code, const std::string& msg) {
    if (ctx) ctx->err = msg;
    return code;
}
int chidg::cuda_fail(chidg_gpu_ctx* ctx, cudaError_t e, const char* what) {
    return fail(ctx, CHIDG_GPU_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}
int chidg::check_launch(chidg_gpu_ctx* ctx, const char* what) {
    ctx->launches++;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(ctx, e, what);
    return CHIDG_GPU_OK;
}
// One stream-ordered memory pool per device for every buffer of the library.
// Allocation and free are ordered on the owning context's stream, so neither
// waits for the device (cudaMalloc / cudaFree synchronise it, which made
// concurrent contexts, e.g. the worker slots of a server, wait for each
// other).  Up to 4 GB of freed memory stays in the pool for the next
// allocations; a stream does not wait on another stream's frees to reuse memory.
static cudaMemPool_t device_pool(int dev) {
    static std::mutex mu;
    static std::map<int, cudaMemPool_t> pools;
    std::lock_guard<std::mutex> lk(mu);
    auto it = pools.find(dev);
    if (it != pools.end()) return it->second;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    // CHIDG_POOL_KEEP_GB: freed memory the pool keeps for reuse (default 4)
    double keep_gb = 4.0;
    if (const char* e = std::getenv("CHIDG_POOL_KEEP_GB")) keep_gb = std::max(0.0, std::atof(e));
    uint64_t keep = (uint64_t)(keep_gb * (double)(1ull << 30));   // the attribute is a 64-bit unsigned value
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    int no = 0;
    cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &no);
    pools[dev] = pool;
    return pool;
}

int chidg::ensure(chidg_gpu_ctx* ctx, Buffer& buf, size_t bytes) {
    if (buf.bytes >= bytes && buf.ptr) return CHIDG_GPU_OK;
    if (buf.ptr) { cudaFreeAsync(buf.ptr, buf.stream); buf.ptr = nullptr; buf.bytes = 0; }
    if (bytes == 0) return CHIDG_GPU_OK;
    cudaMemPool_t pool = device_pool(ctx->device);
    if (!pool) return fail(ctx, CHIDG_GPU_ECUDA, "no stream-ordered memory pool on this device");
    // 256 bytes of slack past the end: bulk copies rounded out to 16-byte
    // boundaries may read up to 15 bytes beyond the last element
    const cudaError_t e = cudaMallocFromPoolAsync(&buf.ptr, bytes + 256, pool, ctx->stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        buf.ptr = nullptr;
        return fail(ctx, CHIDG_GPU_ENOMEM, "device allocation of " + std::to_string(bytes) + " bytes failed");
    }
    buf.bytes = bytes;
    buf.stream = ctx->stream;
    return CHIDG_GPU_OK;
}
void chidg::release(Buffer& buf) {
    if (buf.ptr) cudaFreeAsync(buf.ptr, buf.stream);
    buf.ptr = nullptr;
    buf.bytes = 0;
}
int chidg::grid_for(int64_t n, int threads, int cap) {
    int64_t g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

// CUDA-event timing of kernel classes (chidg_gpu_ctx_set_profiling).
static cudaEvent_t prof_event(chidg_gpu_ctx* ctx) {
    if (!ctx->prof_pool.empty()) {
        cudaEvent_t e = ctx->prof_pool.back();
        ctx->prof_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}
int chidg::prof_begin(chidg_gpu_ctx* ctx, int cls) {
    if (!ctx->profiling) return -1;
    EvPair p{prof_event(ctx), prof_event(ctx), cls};
    cudaEventRecord(p.a, ctx->stream);
    ctx->prof_pending.push_back(p);
    return (int)ctx->prof_pending.size() - 1;
}
void chidg::prof_end(chidg_gpu_ctx* ctx, int h) {
    if (h < 0 || h >= (int)ctx->prof_pending.size()) return;
    cudaEventRecord(ctx->prof_pending[h].b, ctx->stream);
}
void chidg::prof_resolve(chidg_gpu_ctx* ctx) {
    for (auto& p : ctx->prof_pending) {
        float ms = 0.f;
        if (cudaEventSynchronize(p.b) == cudaSuccess && cudaEventElapsedTime(&ms, p.a, p.b) == cudaSuccess) {
            ctx->prof_ms[p.cls] += ms;
            ctx->prof_count[p.cls]++;
        }
        cudaGetLastError();
        ctx->prof_pool.push_back(p.a);
        ctx->prof_pool.push_back(p.b);
    }
    ctx->prof_pending.clear();
}
extern "C" int chidg_gpu_ctx_set_profiling(chidg_gpu_ctx* ctx, int32_t on) {
    if (!ctx) return CHIDG_GPU_EINVAL;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    prof_resolve(ctx);
    for (int c = 0; c < kProfClasses; ++c) { ctx->prof_ms[c] = 0.0; ctx->prof_count[c] = 0; }
    ctx->profiling = on != 0;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_ctx_kernel_time(chidg_gpu_ctx* ctx, int32_t cls, double* total_ms, int64_t* count) {
    if (!ctx || cls < 0 || cls >= kProfClasses || !total_ms || !count) return CHIDG_GPU_EINVAL;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    prof_resolve(ctx);
    *total_ms = ctx->prof_ms[cls];
    *count = ctx->prof_count[cls];
    return CHIDG_GPU_OK;
}

// Status word of the dataflow sweeps, read back as one double slot.
int chidg::status_word(chidg_gpu_ctx* ctx, double slot_value) {
    int w = 0;
    std::memcpy(&w, &slot_value, sizeof(int));
    if (w != 0) return fail(ctx, CHIDG_GPU_ETIMEOUT, "ILU sweep: a bounded wait for a parent row ran out");
    return CHIDG_GPU_OK;
}

// Two-pass reductions into ctx->d_scal[slot..slot+nq).
int chidg::reduce_partials(chidg_gpu_ctx* ctx, const double* partial, int ncta, int nq, int slot, bool do_sqrt) {
    k_reduce_partials<<<1, 1024, 0, ctx->stream>>>(partial, ncta, nq, ctx->d_scal + slot, do_sqrt ? 1 : 0);
    return check_launch(ctx, "k_reduce_partials");
}
int chidg::fetch_scalars(chidg_gpu_ctx* ctx, int slot, int count, double* out) {
    cudaError_t e = cudaMemcpyAsync(ctx->h_scal + slot, ctx->d_scal + slot, sizeof(double) * count, cudaMemcpyDeviceToHost, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "scalar download");
    e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "stream synchronize");
    std::memcpy(out, ctx->h_scal + slot, sizeof(double) * count);
    return CHIDG_GPU_OK;
}
int chidg::push_scalars(chidg_gpu_ctx* ctx, int slot, int count, const double* in) {
    // The pinned staging slots are private to this call: wait for earlier
    // copies out of the same slots before overwriting them.
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "stream synchronize");
    std::memcpy(ctx->h_scal + slot, in, sizeof(double) * count);
    e = cudaMemcpyAsync(ctx->d_scal + slot, ctx->h_scal + slot, sizeof(double) * count, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "scalar upload");
    return CHIDG_GPU_OK;
}

unsigned* chidg::cta_counter(chidg_gpu_ctx* ctx) { return (unsigned*)ctx->d_status + 2; }

// dot products of x with nq vectors y + q*ystride, results in d_scal[slot+q]
template <typename T>
int chidg::mdot(chidg_gpu_ctx* ctx, int64_t n, const T* x, const T* y, int64_t ystride, int nq, int slot, const double* rows,
                int nrow, int row_slot) {
    const int threads = 256;
    const int ncta = grid_for(n, threads, ctx->nsm * 4);
    int st = ensure(ctx, ctx->partial, sizeof(double) * (size_t)ncta * (std::max(nq, 1) + 1));
    if (st) return st;
    k_mdot<T><<<ncta, threads, 0, ctx->stream>>>(n, x, y, ystride, nq, (double*)ctx->partial.ptr, ctx->d_scal + slot, rows,
                                                nrow, ctx->d_scal + row_slot, cta_counter(ctx));
    return check_launch(ctx, "k_mdot");
}
template int chidg::mdot<double>(chidg_gpu_ctx*, int64_t, const double*, const double*, int64_t, int, int, const double*, int, int);
template int chidg::mdot<float>(chidg_gpu_ctx*, int64_t, const float*, const float*, int64_t, int, int, const double*, int, int);

extern "C" int chidg_gpu_ctx_create(int device, void* stream, chidg_gpu_ctx** out) {
    if (!out) return CHIDG_GPU_EINVAL;
    *out = nullptr;
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || device < 0 || device >= ndev) { cudaGetLastError(); return CHIDG_GPU_EINVAL; }
    e = cudaSetDevice(device);
    if (e != cudaSuccess) return CHIDG_GPU_ECUDA;
    auto* ctx = new chidg_gpu_ctx();
    ctx->device = device;
    if (stream) { ctx->stream = (cudaStream_t)stream; ctx->own_stream = false; }
    else {
        e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) { delete ctx; return CHIDG_GPU_ECUDA; }
        ctx->own_stream = true;
    }
    cudaDeviceGetAttribute(&ctx->nsm, cudaDevAttrMultiProcessorCount, device);
    if (cudaMalloc(&ctx->d_status, sizeof(int) * 4) != cudaSuccess ||
        cudaMalloc(&ctx->d_scal, sizeof(double) * kScalSlots) != cudaSuccess ||
        cudaMallocHost(&ctx->h_scal, sizeof(double) * kScalSlots) != cudaSuccess ||
        cudaMallocHost(&ctx->h_status, sizeof(int) * 4) != cudaSuccess) {
        cudaGetLastError();
        chidg_gpu_ctx_destroy(ctx);
        return CHIDG_GPU_ENOMEM;
    }
    // the CTA counter starts at zero (on the stream that uses it)
    if (cudaMemsetAsync(ctx->d_status, 0, sizeof(int) * 4, ctx->stream) != cudaSuccess) {
        cudaGetLastError();
        chidg_gpu_ctx_destroy(ctx);
        return CHIDG_GPU_ECUDA;
    }
    *out = ctx;
    return CHIDG_GPU_OK;
}

extern "C" int chidg_gpu_ctx_destroy(chidg_gpu_ctx* ctx) {
    if (!ctx) return CHIDG_GPU_OK;
    cudaSetDevice(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    prof_resolve(ctx);
    for (cudaEvent_t e : ctx->prof_pool) cudaEventDestroy(e);
    release(ctx->partial);
    release(ctx->partial2);
    for (Workspace* w : {&ctx->ws64, &ctx->ws32})
        for (Buffer* b : {&w->V, &w->Z, &w->x0, &w->zr, &w->dz, &w->tmp, &w->rowsq}) release(*b);
    release(ctx->mix_v32);
    release(ctx->mix_z32);
    release_batch_graphs(ctx);
    for (BatchBuffers* bb : {&ctx->batch, &ctx->batch_inner}) {
        for (Buffer* b : {&bb->cstart, &bb->csys, &bb->sys_chunk, &bb->sys_row, &bb->row_sys, &bb->state, &bb->partial,
                          &bb->rowsq, &bb->out})
            release(*b);
        for (cudaEvent_t& e : bb->ev)
            if (e) cudaEventDestroy(e);
        if (bb->h_count) cudaFreeHost(bb->h_count);
    }
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);   // the frees above are ordered on this stream
    if (ctx->d_status) cudaFree(ctx->d_status);
    if (ctx->d_scal) cudaFree(ctx->d_scal);
    if (ctx->h_scal) cudaFreeHost(ctx->h_scal);
    if (ctx->h_status) cudaFreeHost(ctx->h_status);
    if (ctx->own_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_ctx_sync(chidg_gpu_ctx* ctx) {
    if (!ctx) return CHIDG_GPU_EINVAL;
    cudaSetDevice(ctx->device);
    const cudaError_t e = cudaStreamSynchronize(ctx->stream);
    return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(ctx, e, "stream synchronize");
}
extern "C" int chidg_gpu_last_error(chidg_gpu_ctx* ctx, char* buf, int32_t buflen) {
    if (!ctx || !buf || buflen <= 0) return CHIDG_GPU_EINVAL;
    std::snprintf(buf, (size_t)buflen, "%s", ctx->err.c_str());
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_error_element(chidg_gpu_ctx* ctx, int32_t* elem) {
    if (!ctx || !elem) return CHIDG_GPU_EINVAL;
    *elem = ctx->err_elem;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_launch_count(chidg_gpu_ctx* ctx, int64_t* count) {
    if (!ctx || !count) return CHIDG_GPU_EINVAL;
    *count = ctx->launches;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_host_alloc(size_t bytes, void** out) {
    if (!out) return CHIDG_GPU_EINVAL;
    const cudaError_t e = cudaMallocHost(out, bytes);
    if (e != cudaSuccess) { cudaGetLastError(); *out = nullptr; return CHIDG_GPU_ENOMEM; }
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_host_free(void* p) {
    if (p) cudaFreeHost(p);
    return CHIDG_GPU_OK;
}

// ---------------------------------------------------------------------------
// chidg_matrix_t
// ---------------------------------------------------------------------------
template <typename T>
static int upload_items(chidg_gpu_ctx* ctx, Buffer& buf, const T* v, size_t n) {
    int st = ensure(ctx, buf, std::max<size_t>(sizeof(T) * n, sizeof(T)));
    if (st) return st;
    if (n == 0) return CHIDG_GPU_OK;
    // from pageable memory: staged before the call returns, so v may go
    const cudaError_t e = cudaMemcpyAsync(buf.ptr, v, sizeof(T) * n, cudaMemcpyHostToDevice, ctx->stream);
    return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(ctx, e, "pattern upload");
}
template <typename T>
static int upload_array(chidg_gpu_ctx* ctx, Buffer& buf, const std::vector<T>& v) {
    return upload_items(ctx, buf, v.data(), v.size());
}

// Triangular sweeps: one row per CTA and a dependency chain through the
// rows, so a row must stream its blocks as fast as one SM allows: use up to
// 1024 threads (G = floor(1024 / b) column groups).
// Threads of a one-CTA-per-row launch: enough for G(b) = stripe_groups(cap, b)
// column groups of b threads for every block size b present, in whole warps.
static int launch_dim_for(int cap, const std::vector<int32_t>& sizes) {
    int t = 32;
    std::vector<char> seen(1025, 0);
    for (int32_t b : sizes) {
        const int bb = std::min(std::max((int)b, 1), 1024);
        if (seen[bb]) continue;
        seen[bb] = 1;
        t = std::max(t, ((stripe_groups(cap, bb) * bb + 31) / 32) * 32);
    }
    return std::min(t, 1024);
}

extern "C" int chidg_gpu_matrix_create(chidg_gpu_ctx* ctx, const chidg_gpu_pattern* pat, chidg_gpu_matrix** out) {
    if (!ctx || !pat || !out) return CHIDG_GPU_EINVAL;
    *out = nullptr;
    cudaSetDevice(ctx->device);
    if (pat->nelem <= 0 || pat->ntime <= 0 || pat->nblocks <= 0 || !pat->elem_nvars || !pat->elem_nterms ||
        !pat->blk_row_elem || !pat->blk_row_time || !pat->blk_col_elem || !pat->blk_col_time || !pat->blk_kind)
        return fail(ctx, CHIDG_GPU_EINVAL, "matrix_create: incomplete pattern");
    auto* A = new chidg_gpu_matrix();
    static std::atomic<int64_t> next_uid{1};
    A->uid = next_uid++;
    A->ctx = ctx;
    A->nelem = pat->nelem;
    A->ntime = pat->ntime;
    A->nrow = pat->nelem * pat->ntime;
    A->nvars.assign(pat->elem_nvars, pat->elem_nvars + A->nelem);
    A->nterms.assign(pat->elem_nterms, pat->elem_nterms + A->nelem);
    A->proc.assign(A->nelem, 0);
    if (pat->elem_proc) A->proc.assign(pat->elem_proc, pat->elem_proc + A->nelem);
    A->eoff.resize(A->nelem);
    int64_t off = 0;
    A->max_b = 0;
    for (int e = 0; e < A->nelem; ++e) {
        if (A->nvars[e] <= 0 || A->nterms[e] <= 0 || A->proc[e] < 0) { delete A; return fail(ctx, CHIDG_GPU_EINVAL, "matrix_create: bad element sizes"); }
        A->eoff[e] = off;
        off += (int64_t)A->ntime * A->bsize(e);
        A->max_b = std::max(A->max_b, A->bsize(e));
    }
    if (A->max_b > 1024) { delete A; return fail(ctx, CHIDG_GPU_EINVAL, "matrix_create: block size above 1024"); }
    A->n = off;
    const int64_t nb = pat->nblocks;
    A->nblk = nb;
    A->re.assign(pat->blk_row_elem, pat->blk_row_elem + nb);
    A->rt.assign(pat->blk_row_time, pat->blk_row_time + nb);
    A->ce.assign(pat->blk_col_elem, pat->blk_col_elem + nb);
    A->ct.assign(pat->blk_col_time, pat->blk_col_time + nb);
    A->kind.assign(pat->blk_kind, pat->blk_kind + nb);
    A->voff.resize(nb);
    int64_t v = 0;
    for (int64_t k = 0; k < nb; ++k) {
        if (A->re[k] < 0 || A->re[k] >= A->nelem || A->ce[k] < 0 || A->ce[k] >= A->nelem ||
            A->rt[k] < 0 || A->rt[k] >= A->ntime || A->ct[k] < 0 || A->ct[k] >= A->ntime ||
            A->kind[k] < 0 || A->kind[k] > 3) { delete A; return fail(ctx, CHIDG_GPU_EINVAL, "matrix_create: block index out of range"); }
        if (A->kind[k] == CHIDG_BLK_LOCAL && A->ct[k] != A->rt[k]) { delete A; return fail(ctx, CHIDG_GPU_EINVAL, "matrix_create: LOCAL block across time levels"); }
        A->voff[k] = v;
        v += (int64_t)A->bsize(A->re[k]) * A->bsize(A->ce[k]);
    }
    A->nval = v;
    A->rowblk.assign(A->nrow, {});
    A->lblk.assign(A->nrow, {});
    A->diag.assign(A->nrow, -1);
    for (int kd = 0; kd < 4; ++kd)
        for (int64_t k = 0; k < nb; ++k) {
            if (A->kind[k] != kd) continue;
            const int r = A->row(A->re[k], A->rt[k]);
            A->rowblk[r].push_back((int32_t)k);
            if (kd == CHIDG_BLK_LOCAL) {
                A->lblk[r].push_back((int32_t)k);
                if (A->ce[k] == A->re[k]) {
                    if (A->diag[r] >= 0) { delete A; return fail(ctx, CHIDG_GPU_EINVAL, "matrix_create: two DIAG blocks in a row"); }
                    A->diag[r] = (int32_t)k;
                }
            }
        }
    for (int r = 0; r < A->nrow; ++r)
        if (A->diag[r] < 0) { delete A; return fail(ctx, CHIDG_GPU_EINVAL, "matrix_create: row without DIAG block"); }
    // a pattern listed in the reference's order (per row: lblks, chi_blks,
    // bc_blks, hb_blks) stores each row's blocks one after another
    for (int r = 0; r < A->nrow && A->rows_contiguous; ++r)
        for (size_t q = 1; q < A->rowblk[r].size(); ++q) {
            const int32_t kp = A->rowblk[r][q - 1], k = A->rowblk[r][q];
            if (A->voff[k] != A->voff[kp] + (int64_t)A->bsize(A->re[kp]) * A->bsize(A->ce[kp])) { A->rows_contiguous = false; break; }
        }
    // CSR in row order for the matvec
    std::vector<int64_t> row_ptr(A->nrow + 1), bvoff, bxoff, yoff(A->nrow), dvoff(A->nrow);
    std::vector<int32_t> bnc, rb(A->nrow);
    A->max_row_cols = 0;
    int64_t cur = 0;
    for (int r = 0; r < A->nrow; ++r) {
        const int e = r / A->ntime, t = r % A->ntime;
        row_ptr[r] = cur;
        int cols = 0;
        for (int32_t k : A->rowblk[r]) {
            bvoff.push_back(A->voff[k]);
            bxoff.push_back(A->seg(A->ce[k], A->ct[k]));
            bnc.push_back(A->bsize(A->ce[k]));
            cols += A->bsize(A->ce[k]);
            ++cur;
        }
        A->max_row_cols = std::max(A->max_row_cols, cols);
        yoff[r] = A->seg(e, t);
        rb[r] = A->bsize(e);
        dvoff[r] = A->voff[A->diag[r]];
    }
    row_ptr[A->nrow] = cur;
    int st;
    if ((st = upload_array(ctx, A->d_row_ptr, row_ptr)) || (st = upload_array(ctx, A->d_blk_voff, bvoff)) ||
        (st = upload_array(ctx, A->d_blk_xoff, bxoff)) || (st = upload_array(ctx, A->d_blk_nc, bnc)) ||
        (st = upload_array(ctx, A->d_row_yoff, yoff)) || (st = upload_array(ctx, A->d_row_b, rb)) ||
        (st = upload_array(ctx, A->d_diag_voff, dvoff)) ||
        (st = upload_array(ctx, A->d_elem_nvars, A->nvars)) || (st = upload_array(ctx, A->d_elem_nterms, A->nterms))) {
        chidg_gpu_matrix_destroy(A);
        return st;
    }
    if (*std::min_element(rb.begin(), rb.end()) != A->max_b) {
        // rows by falling cost, for the streamed matvec
        std::vector<int64_t> cost(A->nrow);
        for (int r = 0; r < A->nrow; ++r)
            for (int32_t k : A->rowblk[r]) cost[r] += (int64_t)rb[r] * A->bsize(A->ce[k]);
        std::vector<int32_t> order(A->nrow);
        for (int r = 0; r < A->nrow; ++r) order[r] = r;
        std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return cost[a] > cost[b]; });
        if ((st = upload_array(ctx, A->d_row_order, order))) { chidg_gpu_matrix_destroy(A); return st; }
    }
    if ((st = ensure(ctx, A->val, sizeof(double) * (size_t)A->nval))) { chidg_gpu_matrix_destroy(A); return st; }
    cudaMemsetAsync(A->val.ptr, 0, sizeof(double) * (size_t)A->nval, ctx->stream);
    A->mv_threads = launch_dim_for(MV_GCAP, rb);
    A->stamp = 1;
    *out = A;
    return CHIDG_GPU_OK;
}

extern "C" int chidg_gpu_matrix_destroy(chidg_gpu_matrix* A) {
    if (!A) return CHIDG_GPU_OK;
    cudaSetDevice(A->ctx->device);
    cudaStreamSynchronize(A->ctx->stream);
    for (Buffer* b : {&A->val, &A->val32, &A->val16, &A->d_row_ptr, &A->d_blk_voff, &A->d_blk_xoff, &A->d_blk_nc,
                      &A->d_row_yoff, &A->d_row_b, &A->d_diag_voff, &A->d_elem_nvars, &A->d_elem_nterms, &A->row_sq,
                      &A->d_tr_src, &A->d_tr_dst, &A->d_tr_nr, &A->d_tr_nc, &A->d_mass_off, &A->d_scale_off, &A->d_row_order})
        release(*b);
    if (A->T) chidg_gpu_matrix_destroy(A->T);
    delete A;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_matrix_nvalues(chidg_gpu_matrix* A, int64_t* n) {
    if (!A || !n) return CHIDG_GPU_EINVAL;
    *n = A->nval;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_matrix_nvec(chidg_gpu_matrix* A, int64_t* n) {
    if (!A || !n) return CHIDG_GPU_EINVAL;
    *n = A->n;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_matrix_stamp(chidg_gpu_matrix* A, int64_t* s) {
    if (!A || !s) return CHIDG_GPU_EINVAL;
    *s = A->stamp;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_matrix_upload(chidg_gpu_matrix* A, const double* host) {
    if (!A || !host) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = A->ctx;
    cudaSetDevice(ctx->device);
    cudaError_t e = cudaMemcpyAsync(A->val.ptr, host, sizeof(double) * (size_t)A->nval, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);   // host arrays are only read during the call
    if (e != cudaSuccess) return cuda_fail(ctx, e, "matrix upload");
    A->stamp++;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_matrix_upload_range(chidg_gpu_matrix* A, const double* host, int64_t first, int64_t count) {
    if (!A || (!host && count > 0) || first < 0 || count < 0 || first + count > A->nval) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = A->ctx;
    cudaSetDevice(ctx->device);
    if (count > 0) {
        cudaError_t e = cudaMemcpyAsync((double*)A->val.ptr + first, host, sizeof(double) * (size_t)count,
                                        cudaMemcpyHostToDevice, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "matrix upload_range");
    }
    A->stamp++;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_matrix_upload_blocks(chidg_gpu_matrix* A, const double* const* ptrs) {
    if (!A || !ptrs) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = A->ctx;
    cudaSetDevice(ctx->device);
    double* d = (double*)A->val.ptr;
    for (int64_t k = 0; k < A->nblk; ++k) {
        if (!ptrs[k]) return fail(ctx, CHIDG_GPU_EINVAL, "upload_blocks: null block pointer");
        const size_t bytes = sizeof(double) * (size_t)A->bsize(A->re[k]) * A->bsize(A->ce[k]);
        const cudaError_t e = cudaMemcpyAsync(d + A->voff[k], ptrs[k], bytes, cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "block upload");
    }
    const cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "block upload");
    A->stamp++;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_matrix_upload_device(chidg_gpu_matrix* A, const double* dev) {
    if (!A || !dev) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = A->ctx;
    cudaSetDevice(ctx->device);
    const cudaError_t e = cudaMemcpyAsync(A->val.ptr, dev, sizeof(double) * (size_t)A->nval, cudaMemcpyDeviceToDevice, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "matrix device copy");
    A->stamp++;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_matrix_download(chidg_gpu_matrix* A, double* host) {
    if (!A || !host) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = A->ctx;
    cudaSetDevice(ctx->device);
    cudaError_t e = cudaMemcpyAsync(host, A->val.ptr, sizeof(double) * (size_t)A->nval, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(ctx, e, "matrix download");
}
extern "C" int chidg_gpu_matrix_clear(chidg_gpu_matrix* A) {
    if (!A) return CHIDG_GPU_EINVAL;
    cudaSetDevice(A->ctx->device);
    const cudaError_t e = cudaMemsetAsync(A->val.ptr, 0, sizeof(double) * (size_t)A->nval, A->ctx->stream);
    if (e != cudaSuccess) return cuda_fail(A->ctx, e, "matrix clear");
    A->stamp++;
    return CHIDG_GPU_OK;
}
static int mass_scale_offsets(chidg_gpu_matrix* A);
extern "C" int chidg_gpu_matrix_scale_diagonal(chidg_gpu_matrix* A, const double* mass, const double* scale) {
    if (!A || !mass || !scale) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = A->ctx;
    cudaSetDevice(ctx->device);
    int64_t m = 0, s = 0;
    for (int e = 0; e < A->nelem; ++e) {
        m += (int64_t)A->nterms[e] * A->nterms[e];
        s += A->nvars[e];
    }
    int st = mass_scale_offsets(A);
    if (st) return st;
    const Buffer& dmo = A->d_mass_off;
    const Buffer& dso = A->d_scale_off;
    Buffer dm, ds;
    if ((st = ensure(ctx, dm, sizeof(double) * m)) || (st = ensure(ctx, ds, sizeof(double) * s))) {
        release(dm); release(ds);
        return st;
    }
    cudaMemcpyAsync(dm.ptr, mass, sizeof(double) * m, cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(ds.ptr, scale, sizeof(double) * s, cudaMemcpyHostToDevice, ctx->stream);
    k_scale_diagonal<<<A->nrow, 256, 0, ctx->stream>>>((double*)A->val.ptr, (const int64_t*)A->d_diag_voff.ptr,
                                                      (const int32_t*)A->d_elem_nvars.ptr, (const int32_t*)A->d_elem_nterms.ptr,
                                                      (const int64_t*)dmo.ptr, (const double*)dm.ptr, (const double*)ds.ptr,
                                                      (const int64_t*)dso.ptr, A->ntime);
    st = check_launch(ctx, "k_scale_diagonal");
    cudaStreamSynchronize(ctx->stream);
    release(dm); release(ds);
    if (st) return st;
    A->stamp++;
    return CHIDG_GPU_OK;
}

// the per-element offsets of packed mass matrices and scales (fixed by the pattern)
static int mass_scale_offsets(chidg_gpu_matrix* A) {
    if (A->d_mass_off.ptr) return CHIDG_GPU_OK;
    std::vector<int64_t> moff(A->nelem), soff(A->nelem);
    int64_t mm = 0, ss = 0;
    for (int e = 0; e < A->nelem; ++e) {
        moff[e] = mm; mm += (int64_t)A->nterms[e] * A->nterms[e];
        soff[e] = ss; ss += A->nvars[e];
    }
    int st;
    if ((st = upload_array(A->ctx, A->d_mass_off, moff)) || (st = upload_array(A->ctx, A->d_scale_off, soff))) {
        release(A->d_mass_off); release(A->d_scale_off);
        return st;
    }
    return CHIDG_GPU_OK;
}

extern "C" int chidg_gpu_vector_mass_scale(const chidg_gpu_vector* x, chidg_gpu_vector* y, const double* mass,
                                           const double* scale) {
    if (!x || !y || !mass || !scale || x == y || x->A != y->A) return CHIDG_GPU_EINVAL;
    chidg_gpu_matrix* A = x->A;
    chidg_gpu_ctx* ctx = A->ctx;
    cudaSetDevice(ctx->device);
    int64_t m = 0, s = 0;
    for (int e = 0; e < A->nelem; ++e) {
        m += (int64_t)A->nterms[e] * A->nterms[e];
        s += A->nvars[e];
    }
    int st = mass_scale_offsets(A);
    if (st) return st;
    Buffer dm, ds;
    if ((st = ensure(ctx, dm, sizeof(double) * m)) || (st = ensure(ctx, ds, sizeof(double) * s))) {
        release(dm); release(ds);
        return st;
    }
    cudaMemcpyAsync(dm.ptr, mass, sizeof(double) * m, cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(ds.ptr, scale, sizeof(double) * s, cudaMemcpyHostToDevice, ctx->stream);
    k_mass_scale<<<A->nrow, 128, 0, ctx->stream>>>((const double*)x->buf.ptr, (double*)y->buf.ptr,
                                                  (const int64_t*)A->d_row_yoff.ptr, (const int32_t*)A->d_elem_nvars.ptr,
                                                  (const int32_t*)A->d_elem_nterms.ptr, (const int64_t*)A->d_mass_off.ptr,
                                                  (const double*)dm.ptr, (const double*)ds.ptr,
                                                  (const int64_t*)A->d_scale_off.ptr, A->ntime);
    st = check_launch(ctx, "k_mass_scale");
    cudaStreamSynchronize(ctx->stream);
    release(dm); release(ds);
    return st;
}

// ---------------------------------------------------------------------------
// chidg_matrix_t%transposed
// ---------------------------------------------------------------------------
// A^T as a matrix of its own: block (c, r) of the same kind for every block
// (r, c) of A.  Row r of A^T lists, per kind, the blocks whose transposed
// partner sits in row r of A, in A's order, then the others by block id; so a
// structurally symmetric pattern (every box mesh, harmonic-balance blocks
// included) gives A^T the block order and value offsets of A.
static int build_transposed(chidg_gpu_matrix* A) {
    chidg_gpu_ctx* ctx = A->ctx;
    const int64_t nb = A->nblk;
    const uint64_t nrow = (uint64_t)A->nrow;
    auto key = [nrow](int r, int c, int kd) { return ((uint64_t)r * nrow + (uint64_t)c) * 4u + (uint64_t)kd; };
    std::unordered_map<uint64_t, int> pos;          // (row, column row, kind) -> position in A's row
    pos.reserve((size_t)nb * 2);
    for (int r = 0; r < A->nrow; ++r)
        for (size_t q = 0; q < A->rowblk[r].size(); ++q) {
            const int32_t k = A->rowblk[r][q];
            pos[key(r, A->row(A->ce[k], A->ct[k]), A->kind[k])] = (int)q;
        }
    struct TB { int row, kind; int64_t order, src; };
    std::vector<TB> tb((size_t)nb);
    for (int64_t k = 0; k < nb; ++k) {
        const int r = A->row(A->ce[k], A->ct[k]);
        const auto it = pos.find(key(r, A->row(A->re[k], A->rt[k]), A->kind[k]));
        tb[k] = {r, A->kind[k], it != pos.end() ? (int64_t)it->second : (int64_t)A->rowblk[r].size() + k, k};
    }
    std::sort(tb.begin(), tb.end(), [](const TB& a, const TB& b) {
        return a.row != b.row ? a.row < b.row : a.kind != b.kind ? a.kind < b.kind : a.order < b.order;
    });
    std::vector<int32_t> bre(nb), brt(nb), bce(nb), bct(nb), bk(nb);
    std::vector<int64_t> src(nb);
    for (int64_t i = 0; i < nb; ++i) {
        const int64_t k = tb[i].src;
        bre[i] = A->ce[k]; brt[i] = A->ct[k]; bce[i] = A->re[k]; bct[i] = A->rt[k]; bk[i] = A->kind[k];
        src[i] = A->voff[k];
    }
    chidg_gpu_pattern pt{};
    pt.nelem = A->nelem; pt.ntime = A->ntime;
    pt.elem_nvars = A->nvars.data(); pt.elem_nterms = A->nterms.data(); pt.elem_proc = A->proc.data();
    pt.nblocks = nb;
    pt.blk_row_elem = bre.data(); pt.blk_row_time = brt.data();
    pt.blk_col_elem = bce.data(); pt.blk_col_time = bct.data(); pt.blk_kind = bk.data();
    chidg_gpu_matrix* T = nullptr;
    int st = chidg_gpu_matrix_create(ctx, &pt, &T);
    if (st) return st;
    std::vector<int64_t> dst(nb);
    std::vector<int32_t> tnr(nb), tnc(nb);
    for (int64_t i = 0; i < nb; ++i) { dst[i] = T->voff[i]; tnr[i] = T->bsize(T->re[i]); tnc[i] = T->bsize(T->ce[i]); }
    if ((st = upload_array(ctx, A->d_tr_src, src)) || (st = upload_array(ctx, A->d_tr_dst, dst)) ||
        (st = upload_array(ctx, A->d_tr_nr, tnr)) || (st = upload_array(ctx, A->d_tr_nc, tnc))) {
        chidg_gpu_matrix_destroy(T);
        return st;
    }
    A->T = T;
    A->T_src_stamp = -1;
    return CHIDG_GPU_OK;
}

extern "C" int chidg_gpu_matrix_set_transposed(chidg_gpu_matrix* A, int32_t transposed) {
    if (!A) return CHIDG_GPU_EINVAL;
    cudaSetDevice(A->ctx->device);
    if (transposed && !A->T) {
        const int st = build_transposed(A);
        if (st) return st;
    }
    A->transposed = transposed != 0;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_matrix_get_transposed(chidg_gpu_matrix* A, int32_t* transposed) {
    if (!A || !transposed) return CHIDG_GPU_EINVAL;
    *transposed = A->transposed ? 1 : 0;
    return CHIDG_GPU_OK;
}

int chidg::matrix_op(chidg_gpu_matrix* A, chidg_gpu_matrix** out) {
    if (!A->transposed) { *out = A; return CHIDG_GPU_OK; }
    chidg_gpu_matrix* T = A->T;
    if (A->T_src_stamp != A->stamp) {
        chidg_gpu_ctx* ctx = A->ctx;
        const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(T->nblk, (int64_t)ctx->nsm * 16));
        k_block_transpose<<<grid, dim3(32, 8), 0, ctx->stream>>>((const double*)A->val.ptr, (double*)T->val.ptr,
                                                                (const int64_t*)A->d_tr_src.ptr, (const int64_t*)A->d_tr_dst.ptr,
                                                                (const int32_t*)A->d_tr_nr.ptr, (const int32_t*)A->d_tr_nc.ptr,
                                                                T->nblk);
        const int st = check_launch(ctx, "k_block_transpose");
        if (st) return st;
        A->T_src_stamp = A->stamp;
        T->stamp = A->stamp;           // the FP32 / BF16 copies of T follow A's stamp
    }
    *out = T;
    return CHIDG_GPU_OK;
}

// Low-precision copies of A for the mixed-precision inner solves.
int chidg::matrix_lowp(chidg_gpu_matrix* A, int precision) {
    chidg_gpu_ctx* ctx = A->ctx;
    if (precision == CHIDG_GPU_FP64) return CHIDG_GPU_OK;
    if (precision == CHIDG_GPU_MIXED_PRECON_FP32) precision = CHIDG_GPU_MIXED_FP32;   // the same FP32 copy
    const int grid = grid_for(A->nval, 256, ctx->nsm * 8);
    int st;
    if (precision == CHIDG_GPU_MIXED_FP32) {
        if (A->val32_stamp == A->stamp) return CHIDG_GPU_OK;
        if ((st = ensure(ctx, A->val32, sizeof(float) * (size_t)A->nval))) return st;
        k_convert<double, float><<<grid, 256, 0, ctx->stream>>>(A->nval, (const double*)A->val.ptr, (float*)A->val32.ptr);
        if ((st = check_launch(ctx, "k_convert A->fp32"))) return st;
        A->val32_stamp = A->stamp;
    } else {
        if (A->val16_stamp == A->stamp) return CHIDG_GPU_OK;
        if ((st = ensure(ctx, A->val16, sizeof(__nv_bfloat16) * (size_t)A->nval))) return st;
        k_convert<double, __nv_bfloat16><<<grid, 256, 0, ctx->stream>>>(A->nval, (const double*)A->val.ptr, (__nv_bfloat16*)A->val16.ptr);
        if ((st = check_launch(ctx, "k_convert A->bf16"))) return st;
        A->val16_stamp = A->stamp;
    }
    return CHIDG_GPU_OK;
}

// y = alpha * A x + beta * z, optional per-row sums of squares of y.  The
// streamed kernel reads each row as one strip of values; rows whose blocks are
// not stored one after another, and blocks over 1024 rows, take the
// one-CTA-per-row kernel, which addresses every block by its own offset.
// CHIDG_MATVEC_ROWS=1 selects the one-CTA-per-row matvec (comparison runs)
static bool matvec_rows_env() {
    static const bool v = [] {
        const char* e = std::getenv("CHIDG_MATVEC_ROWS");
        return e && e[0] == '1';
    }();
    return v;
}

template <typename TA, typename TV>
int chidg::matvec_launch(chidg_gpu_matrix* A, const TA* val, const TV* x, TV* y, const TV* z, double alpha, double beta, double* row_sq) {
    chidg_gpu_ctx* ctx = A->ctx;
    using ACC = typename AccOf<TV>::type;
    const int ph = prof_begin(ctx, sizeof(TA) == 8 ? kProfMatvec : kProfMatvec32);
    if (A->max_b <= SS_MAX_B && A->rows_contiguous && !matvec_rows_env()) {
        // streamed: persistent CTAs, row values prefetched by bulk copies
        const StreamShape sh = stream_shape_for(kShapeMatvec, A->max_b, (int)sizeof(TA));
        MatvecRows R{(const int64_t*)A->d_row_ptr.ptr, (const int64_t*)A->d_blk_voff.ptr, (const int64_t*)A->d_blk_xoff.ptr,
                     (const int32_t*)A->d_blk_nc.ptr, (const int64_t*)A->d_row_yoff.ptr, (const int32_t*)A->d_row_b.ptr};
        if ((size_t)sh.stage_bytes < (size_t)A->max_b * sizeof(TA) + 16)
            return fail(ctx, CHIDG_GPU_EINVAL, "streamed matvec: stage smaller than one block column");
        auto launch = [&](auto k, int cw) -> int {
            const size_t smem = matvec_stream_smem(sizeof(ACC), sh.nstage, sh.stage_bytes, A->max_row_cols, 32 * cw);
            int st2;
            if ((st2 = raise_smem_limit((const void*)k, smem))) return fail(ctx, st2, "streamed matvec shared memory");
            const int per_sm = resident_ctas((const void*)k, 32 * cw + 32, smem);
            if (per_sm < 1) return fail(ctx, CHIDG_GPU_EINVAL, "streamed matvec: shape does not fit an SM");
            const int grid = std::max(1, std::min(A->nrow, per_sm * ctx->nsm));
            const RowMask mk = ctx->row_mask.nrow == A->nrow ? ctx->row_mask : RowMask{};
            k<<<grid, 32 * cw + 32, smem, ctx->stream>>>(R, A->nrow, val, x, y, z, alpha, beta, row_sq,
                                                         (int*)(ctx->d_scal + kSlotStatus), kSpinLimit, sh.nstage,
                                                         sh.stage_bytes, A->max_row_cols, mk, (const int32_t*)A->d_row_order.ptr);
            return CHIDG_GPU_OK;
        };
        int st2;
        switch (sh.cw) {
            case 16: st2 = launch(k_matvec_stream<TA, TV, ACC, 16>, 16); break;
            case 4: st2 = launch(k_matvec_stream<TA, TV, ACC, 4>, 4); break;
            default: st2 = launch(k_matvec_stream<TA, TV, ACC, 8>, 8);
        }
        if (st2) return st2;
    } else {
        const size_t smem = sizeof(ACC) * ((size_t)A->max_row_cols + A->mv_threads) + 512;
        const int st2 = set_matvec_smem(A);
        if (st2) return fail(ctx, st2, "matvec shared memory");
        k_matvec<TA, TV, TV, ACC><<<A->nrow, A->mv_threads, smem, ctx->stream>>>(
            val, (const int64_t*)A->d_row_ptr.ptr, (const int64_t*)A->d_blk_voff.ptr, (const int64_t*)A->d_blk_xoff.ptr,
            (const int32_t*)A->d_blk_nc.ptr, (const int64_t*)A->d_row_yoff.ptr, (const int32_t*)A->d_row_b.ptr, x, y, z, alpha, beta, row_sq);
    }
    prof_end(ctx, ph);
    return check_launch(ctx, "k_matvec");
}
template int chidg::matvec_launch<double, double>(chidg_gpu_matrix*, const double*, const double*, double*, const double*, double, double, double*);
template int chidg::matvec_launch<float, float>(chidg_gpu_matrix*, const float*, const float*, float*, const float*, double, double, double*);
template int chidg::matvec_launch<__nv_bfloat16, float>(chidg_gpu_matrix*, const __nv_bfloat16*, const float*, float*, const float*, double, double, double*);

int chidg::raise_smem_limit(const void* func, size_t bytes) {
    if (bytes <= 48 * 1024) return CHIDG_GPU_OK;
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> limit;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    size_t& cur = limit[{dev, func}];
    if (bytes <= cur) return CHIDG_GPU_OK;
    const cudaError_t e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return CHIDG_GPU_ECUDA;
    }
    cur = bytes;
    return CHIDG_GPU_OK;
}

int chidg::set_matvec_smem(chidg_gpu_matrix* A) {
    // allow > 48 KB dynamic shared memory when a row has many wide blocks
    const size_t smem = sizeof(double) * ((size_t)A->max_row_cols + A->mv_threads) + 512;
    int st;
    if ((st = raise_smem_limit((const void*)k_matvec<double, double, double, double>, smem)) ||
        (st = raise_smem_limit((const void*)k_matvec<float, float, float, float>, smem)) ||
        (st = raise_smem_limit((const void*)k_matvec<__nv_bfloat16, float, float, float>, smem)))
        return st;
    return CHIDG_GPU_OK;
}

// ---------------------------------------------------------------------------
// chidg_vector_t
// ---------------------------------------------------------------------------
extern "C" int chidg_gpu_vector_create(chidg_gpu_matrix* A, chidg_gpu_vector** out) {
    if (!A || !out) return CHIDG_GPU_EINVAL;
    *out = nullptr;
    chidg_gpu_ctx* ctx = A->ctx;
    cudaSetDevice(ctx->device);
    auto* x = new chidg_gpu_vector();
    x->A = A;
    x->ctx = ctx;
    x->n = A->n;
    int st = ensure(ctx, x->buf, sizeof(double) * (size_t)x->n);
    if (st) { delete x; return st; }
    cudaMemsetAsync(x->buf.ptr, 0, sizeof(double) * (size_t)x->n, ctx->stream);
    // the buffer is stream-ordered on ctx->stream; callers may use its device
    // pointer (chidg_gpu_vector_device_ptr) on streams of their own
    cudaStreamSynchronize(ctx->stream);
    *out = x;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_vector_destroy(chidg_gpu_vector* x) {
    if (!x) return CHIDG_GPU_OK;
    cudaSetDevice(x->ctx->device);
    cudaStreamSynchronize(x->ctx->stream);
    release(x->buf);
    delete x;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_vector_upload(chidg_gpu_vector* x, const double* host) {
    if (!x || !host) return CHIDG_GPU_EINVAL;
    cudaSetDevice(x->ctx->device);
    cudaError_t e = cudaMemcpyAsync(x->buf.ptr, host, sizeof(double) * (size_t)x->n, cudaMemcpyHostToDevice, x->ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(x->ctx->stream);
    return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(x->ctx, e, "vector upload");
}
extern "C" int chidg_gpu_vector_upload_range(chidg_gpu_vector* x, const double* host, int64_t first, int64_t count) {
    if (!x || (!host && count > 0) || first < 0 || count < 0 || first + count > x->n) return CHIDG_GPU_EINVAL;
    cudaSetDevice(x->ctx->device);
    if (count == 0) return CHIDG_GPU_OK;
    cudaError_t e = cudaMemcpyAsync((double*)x->buf.ptr + first, host, sizeof(double) * (size_t)count,
                                    cudaMemcpyHostToDevice, x->ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(x->ctx->stream);
    return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(x->ctx, e, "vector upload_range");
}
extern "C" int chidg_gpu_vector_download(chidg_gpu_vector* x, double* host) {
    if (!x || !host) return CHIDG_GPU_EINVAL;
    cudaSetDevice(x->ctx->device);
    cudaError_t e = cudaMemcpyAsync(host, x->buf.ptr, sizeof(double) * (size_t)x->n, cudaMemcpyDeviceToHost, x->ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(x->ctx->stream);
    return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(x->ctx, e, "vector download");
}
extern "C" int chidg_gpu_vector_upload_device(chidg_gpu_vector* x, const double* dev) {
    if (!x || !dev) return CHIDG_GPU_EINVAL;
    cudaSetDevice(x->ctx->device);
    const cudaError_t e = cudaMemcpyAsync(x->buf.ptr, dev, sizeof(double) * (size_t)x->n, cudaMemcpyDeviceToDevice, x->ctx->stream);
    return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(x->ctx, e, "vector device copy");
}
extern "C" int chidg_gpu_vector_device_ptr(chidg_gpu_vector* x, double** dev) {
    if (!x || !dev) return CHIDG_GPU_EINVAL;
    *dev = (double*)x->buf.ptr;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_vector_clear(chidg_gpu_vector* x) {
    if (!x) return CHIDG_GPU_EINVAL;
    cudaSetDevice(x->ctx->device);
    const cudaError_t e = cudaMemsetAsync(x->buf.ptr, 0, sizeof(double) * (size_t)x->n, x->ctx->stream);
    return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(x->ctx, e, "vector clear");
}
extern "C" int chidg_gpu_vector_copy(chidg_gpu_vector* dst, const chidg_gpu_vector* src) {
    if (!dst || !src || dst->n != src->n) return CHIDG_GPU_EINVAL;
    cudaSetDevice(dst->ctx->device);
    const cudaError_t e = cudaMemcpyAsync(dst->buf.ptr, src->buf.ptr, sizeof(double) * (size_t)dst->n, cudaMemcpyDeviceToDevice, dst->ctx->stream);
    return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(dst->ctx, e, "vector copy");
}
extern "C" int chidg_gpu_vector_axpy(chidg_gpu_vector* y, double a, const chidg_gpu_vector* x) {
    if (!y || !x || y->n != x->n) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = y->ctx;
    cudaSetDevice(ctx->device);
    k_axpby<double, double><<<grid_for(y->n, 256, ctx->nsm * 8), 256, 0, ctx->stream>>>(y->n, a, nullptr, (const double*)x->buf.ptr, 1.0, (double*)y->buf.ptr);
    return check_launch(ctx, "k_axpby");
}
extern "C" int chidg_gpu_vector_scale(chidg_gpu_vector* x, double a) {
    if (!x) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = x->ctx;
    cudaSetDevice(ctx->device);
    k_axpby<double, double><<<grid_for(x->n, 256, ctx->nsm * 8), 256, 0, ctx->stream>>>(x->n, a, nullptr, (const double*)x->buf.ptr, 0.0, (double*)x->buf.ptr);
    return check_launch(ctx, "k_axpby");
}
extern "C" int chidg_gpu_vector_dot(const chidg_gpu_vector* x, const chidg_gpu_vector* y, double* out) {
    if (!x || !y || !out || x->n != y->n) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = x->ctx;
    cudaSetDevice(ctx->device);
    int st = mdot<double>(ctx, x->n, (const double*)x->buf.ptr, (const double*)y->buf.ptr, 0, 1, kSlotTmp);
    if (st) return st;
    return fetch_scalars(ctx, kSlotTmp, 1, out);
}
extern "C" int chidg_gpu_vector_norm(const chidg_gpu_vector* x, double* out) {
    if (!x || !out) return CHIDG_GPU_EINVAL;
    double s;
    int st = chidg_gpu_vector_dot(x, x, &s);
    if (st) return st;
    *out = std::sqrt(s);
    return CHIDG_GPU_OK;
}
// Failure detection without a fault: the bounded waits of the streamed
// kernels (a flag another CTA sets, an mbarrier the producer completes) are
// made to run out on a flag that nothing sets and an mbarrier that nobody
// arrives at.  Each gives up after `limit` clock cycles and reports it:
// bit 0 the flag wait, bit 1 the mbarrier wait.  One thread, one CTA.
static __global__ void k_bounded_wait_selftest(const unsigned* flag, long long limit, int* bits) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    int b = 0;
    if (!wait_flag(flag, 0, 1u, limit)) b |= 1;
    if (!mbar_wait(&bar, 0u, limit)) b |= 2;
    *bits = b;
}

extern "C" int chidg_gpu_selftest_bounded_waits(chidg_gpu_ctx* ctx, int64_t limit_cycles, int32_t* bits) {
    if (!ctx || !bits || limit_cycles <= 0 || limit_cycles > 4000000000LL) return CHIDG_GPU_EINVAL;
    cudaSetDevice(ctx->device);
    Buffer flag, out;
    int st;
    if ((st = ensure(ctx, flag, 64)) || (st = ensure(ctx, out, sizeof(int)))) { release(flag); release(out); return st; }
    cudaMemsetAsync(flag.ptr, 0, 64, ctx->stream);
    k_bounded_wait_selftest<<<1, 32, 0, ctx->stream>>>((const unsigned*)flag.ptr, (long long)limit_cycles, (int*)out.ptr);
    st = check_launch(ctx, "k_bounded_wait_selftest");
    int h = 0;
    if (!st) {
        cudaError_t e = cudaMemcpyAsync(&h, out.ptr, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) st = cuda_fail(ctx, e, "bounded wait self-test");
    }
    release(flag);
    release(out);
    *bits = h;
    return st;
}

// chidg_vector%norm_fields (type_chidg_vector.f90:1319-1352): per field the
// L2 norm over all elements, time levels and modes.  Every element must have
// nfields fields.
extern "C" int chidg_gpu_vector_norm_fields(const chidg_gpu_vector* x, double* out, int32_t nfields) {
    if (!x || !out || nfields <= 0 || nfields > 32) return CHIDG_GPU_EINVAL;
    chidg_gpu_matrix* A = x->A;
    chidg_gpu_ctx* ctx = x->ctx;
    cudaSetDevice(ctx->device);
    for (int e = 0; e < A->nelem; ++e)
        if (A->nvars[e] != nfields) return fail(ctx, CHIDG_GPU_EINVAL, "norm_fields: an element with another field count");
    const int grid = std::max(1, std::min(A->nrow, ctx->nsm * 4));
    int st = ensure(ctx, ctx->partial2, sizeof(double) * (size_t)grid * nfields);
    if (st) return st;
    k_field_sumsq<<<grid, 256, 0, ctx->stream>>>((const double*)x->buf.ptr, (const int64_t*)A->d_row_yoff.ptr,
                                                (const int32_t*)A->d_elem_nterms.ptr, A->nrow, A->ntime, nfields,
                                                (double*)ctx->partial2.ptr);
    if ((st = check_launch(ctx, "k_field_sumsq"))) return st;
    if ((st = reduce_partials(ctx, (const double*)ctx->partial2.ptr, grid, nfields, kSlotFields, true))) return st;
    return fetch_scalars(ctx, kSlotFields, nfields, out);
}

extern "C" int chidg_gpu_matvec(chidg_gpu_matrix* A, const chidg_gpu_vector* x, chidg_gpu_vector* y) {
    if (!A || !x || !y || x->n != A->n || y->n != A->n || x == y) return CHIDG_GPU_EINVAL;
    cudaSetDevice(A->ctx->device);
    chidg_gpu_matrix* S;                 // A, or A^T when A->transposed (operator_chidg_mv.f90:46-60)
    int st = matrix_op(A, &S);
    if (st) return st;
    return matvec_launch<double, double>(S, (const double*)S->val.ptr, (const double*)x->buf.ptr, (double*)y->buf.ptr,
                                         nullptr, 1.0, 0.0, nullptr);
}

// ---------------------------------------------------------------------------
// Preconditioner programmes
// ---------------------------------------------------------------------------
namespace {

// the FP32 factorisation's tensor-core kernels take blocks of up to this size
constexpr int FACTOR32_SMALL = 136;

// transposed LOCAL block: first LOCAL block of row (p,t) whose column is e
// (type_domain_matrix.f90:592-627)
int find_trans(const chidg_gpu_matrix* A, int p, int t, int e) {
    for (int32_t kk : A->lblk[A->row(p, t)])
        if (A->ce[kk] == e) return kk;
    return -1;
}

}  // namespace

// ILU0 / Jacobi on a single rank: one programme row per matrix row.
static int build_ilu0(const chidg_gpu_matrix* A, bool jacobi, IluProgram& P, std::string& err) {
    P = IluProgram();
    P.diagonal = jacobi;
    P.n_ext = A->n;
    P.nlocal_rows = A->nrow;
    // programme row id == matrix row id (e*ntime+t)
    for (int r = 0; r < A->nrow; ++r) {
        const int e = r / A->ntime, t = r % A->ntime;
        P.prow_b.push_back(A->bsize(e));
        P.prow_elem.push_back(e);
        P.v_off.push_back(A->seg(e, t));
        P.z_off.push_back(A->seg(e, t));
        P.diagA_off.push_back(A->voff[A->diag[r]]);
        P.diag_blk.push_back(A->diag[r]);
        P.lo.emplace_back();
        P.up.emplace_back();
    }
    if (jacobi) return CHIDG_GPU_OK;
    for (int r = 0; r < A->nrow; ++r) {
        const int e = r / A->ntime, t = r % A->ntime;
        for (int32_t k : A->lblk[r]) {
            const int p = A->ce[k];
            if (p < e) {   // type_domain_matrix.f90:295-302, single rank
                const int kt = find_trans(A, p, t, e);
                if (kt < 0) { err = "ilu0: no transposed block found"; return CHIDG_GPU_EINVAL; }
                IluEntry en;
                en.parent = A->row(p, t);
                en.a_off = A->voff[k];
                en.t_off = A->voff[kt];
                en.nc = A->bsize(p);
                en.blk = k;
                P.lo[r].push_back(en);
            } else if (p > e) {
                IluEntry en;
                en.parent = A->row(p, t);
                en.a_off = A->voff[k];
                en.nc = A->bsize(p);
                en.blk = k;
                P.up[r].push_back(en);
            }
        }
    }
    return CHIDG_GPU_OK;
}

// precon_HB (precon_HB.f90:169-310): one programme row per element over all
// its time levels (the element's segment is contiguous: time-major inside the
// element).  Its D is assembled, not factored: the DIAG block of level t at
// (t, t), the hb_blks block of row (e, ta) and column (e, tb) at (ta, tb) (it
// holds D(ta,tb) mass per field, what the reference places there), zero
// elsewhere; then inverted.  No lower or upper entries.
static int build_hb(const chidg_gpu_matrix* A, IluProgram& P, std::string& err) {
    P = IluProgram();
    P.n_ext = A->n;
    P.nlocal_rows = A->nelem;
    P.assembled = true;
    P.diagonal = true;
    P.asm_ptr.assign(1, 0);
    for (int e = 0; e < A->nelem; ++e) {
        const int b = A->bsize(e), B = b * A->ntime;
        if (B > 1024) { err = "precon_HB: element block over all time levels above 1024 rows"; return CHIDG_GPU_EINVAL; }
        P.prow_b.push_back(B);
        P.prow_elem.push_back(e);
        P.v_off.push_back(A->eoff[e]);
        P.z_off.push_back(A->eoff[e]);
        P.diagA_off.push_back(-1);
        P.diag_blk.push_back(-1);
        P.lo.emplace_back();
        P.up.emplace_back();
        auto piece = [&](int32_t k, int ta, int tb) {
            P.asm_src.push_back(A->voff[k]);
            P.asm_r0.push_back(ta * b);
            P.asm_c0.push_back(tb * b);
            P.asm_nr.push_back(b);
            P.asm_nc.push_back(b);
        };
        for (int ta = 0; ta < A->ntime; ++ta) {
            const int r = A->row(e, ta);
            piece(A->diag[r], ta, ta);
            for (int32_t k : A->rowblk[r])
                if (A->kind[k] == CHIDG_BLK_HB && A->ce[k] == e && A->ct[k] != ta) piece(k, ta, A->ct[k]);
        }
        P.asm_ptr.push_back((int32_t)P.asm_src.size());
    }
    return CHIDG_GPU_OK;
}

// RAS+ILU0: subdomain s plays MPI rank s.  Local rows in local element order,
// then the overlap rows received from each neighbour rank, as the reference
// builds them (RASILU0/type_RASILU0_send_comm.f90:66-275 selects the sent
// blocks, RASILU0/type_RASILU0_recv_dom_comm.f90:59-305 classifies them).
static int build_rasilu0(const chidg_gpu_matrix* A, IluProgram& P, std::string& err) {
    P = IluProgram();
    P.subdomains = true;
    if (A->ntime != 1) { err = "rasilu0: single time level only"; return CHIDG_GPU_EINVAL; }
    int nsub = 0;
    for (int e = 0; e < A->nelem; ++e) nsub = std::max(nsub, A->proc[e] + 1);
    std::vector<std::vector<int>> elems(nsub);
    std::vector<int> lidx(A->nelem);
    for (int e = 0; e < A->nelem; ++e) { lidx[e] = (int)elems[A->proc[e]].size(); elems[A->proc[e]].push_back(e); }
    // does element f (owned by q) have a face neighbour on rank s?
    auto touches = [&](int f, int s) {
        for (int32_t k : A->lblk[A->row(f, 0)])
            if (A->ce[k] != f && A->proc[A->ce[k]] == s) return true;
        return false;
    };
    int64_t ov_cursor = A->n;
    P.nlocal_rows = 0;
    for (int s = 0; s < nsub; ++s) {
        // local rows
        std::vector<int> local_prow(elems[s].size());
        for (size_t i = 0; i < elems[s].size(); ++i) {
            const int e = elems[s][i];
            const int pr = (int)P.prow_b.size();
            local_prow[i] = pr;
            P.prow_b.push_back(A->bsize(e));
            P.prow_elem.push_back(e);
            P.v_off.push_back(A->seg(e, 0));
            P.z_off.push_back(A->seg(e, 0));
            P.diagA_off.push_back(A->voff[A->diag[A->row(e, 0)]]);
            P.diag_blk.push_back(A->diag[A->row(e, 0)]);
            P.lo.emplace_back();
            P.up.emplace_back();
            P.nlocal_rows++;
        }
        // overlap rows, per neighbour rank in order of first appearance
        std::vector<int> comm;
        for (int e : elems[s])
            for (int32_t k : A->lblk[A->row(e, 0)]) {
                const int pp = A->proc[A->ce[k]];
                if (pp != s && std::find(comm.begin(), comm.end(), pp) == comm.end()) comm.push_back(pp);
            }
        std::map<int, int> ov_prow;   // element -> overlap programme row (unique per subdomain)
        struct OvInfo { int f; int pr; std::vector<int32_t> lower_blk, upper_blk; };
        std::vector<std::vector<OvInfo>> ovs(comm.size());
        for (size_t ic = 0; ic < comm.size(); ++ic) {
            const int q = comm[ic];
            for (int f : elems[q]) {
                if (!touches(f, s)) continue;
                const int pr = (int)P.prow_b.size();
                P.prow_b.push_back(A->bsize(f));
                P.prow_elem.push_back(f);
                P.v_off.push_back(A->seg(f, 0));      // halo of v
                P.z_off.push_back(ov_cursor);
                ov_cursor += A->bsize(f);
                P.diagA_off.push_back(A->voff[A->diag[A->row(f, 0)]]);
                P.diag_blk.push_back(-1);
                P.lo.emplace_back();
                P.up.emplace_back();
                ov_prow[f] = pr;
                OvInfo oi;
                oi.f = f;
                oi.pr = pr;
                // received blocks: (1) coupling to rank s, (2) coupling to other sent
                // neighbours on q; the diagonal is handled separately
                std::vector<int32_t> recv;
                for (int32_t k : A->lblk[A->row(f, 0)])
                    if (A->ce[k] != f && A->proc[A->ce[k]] == s) recv.push_back(k);
                for (int32_t k : A->lblk[A->row(f, 0)]) {
                    const int nb = A->ce[k];
                    if (nb == f || A->proc[nb] != q) continue;
                    if (touches(nb, s)) recv.push_back(k);
                }
                for (int32_t k : recv) {
                    const int par = A->ce[k];
                    if (A->proc[par] == s) oi.lower_blk.push_back(k);     // coupled to the receiver: lower
                    else if (par < f) oi.lower_blk.push_back(k);          // same owner, lower local index
                    else if (par > f) oi.upper_blk.push_back(k);
                }
                ovs[ic].push_back(oi);
            }
        }
        // local entries (type_domain_matrix.f90:295-302 with rank s)
        for (size_t i = 0; i < elems[s].size(); ++i) {
            const int e = elems[s][i];
            const int pr = local_prow[i];
            for (int32_t k : A->lblk[A->row(e, 0)]) {
                const int p = A->ce[k];
                if (p == e) continue;
                const int pp = A->proc[p];
                const bool lo = (pp == s && lidx[p] < (int)i) || (pp < s);
                const bool up = (pp == s && lidx[p] > (int)i) || (pp > s);
                if (lo) {
                    if (pp != s) continue;   // parent_proc /= IRANK: skipped by factor and forward sweep
                    if (i == 0) continue;    // the factor loop starts at the second row
                    const int kt = find_trans(A, p, 0, e);
                    if (kt < 0) { err = "rasilu0: no transposed block found"; return CHIDG_GPU_EINVAL; }
                    IluEntry en;
                    en.parent = local_prow[lidx[p]];
                    en.a_off = A->voff[k];
                    en.t_off = A->voff[kt];
                    en.nc = A->bsize(p);
                    en.blk = k;
                    P.lo[pr].push_back(en);
                } else if (up) {
                    IluEntry en;
                    if (pp == s) en.parent = local_prow[lidx[p]];
                    else {
                        auto it = ov_prow.find(p);
                        if (it == ov_prow.end()) { err = "rasilu0: upper block to an element outside the overlap"; return CHIDG_GPU_EINVAL; }
                        en.parent = it->second;
                    }
                    en.a_off = A->voff[k];
                    en.nc = A->bsize(p);
                    en.blk = k;
                    P.up[pr].push_back(en);
                }
            }
        }
        // overlap entries
        for (auto& O : ovs)
            for (auto& oi : O) {
                for (int32_t k : oi.lower_blk) {
                    const int par = A->ce[k];
                    const int kt = find_trans(A, par, 0, oi.f);
                    if (kt < 0) { err = "rasilu0: no transposed block found for overlap block"; return CHIDG_GPU_EINVAL; }
                    IluEntry en;
                    if (A->proc[par] == s) en.parent = local_prow[lidx[par]];
                    else {
                        auto it = ov_prow.find(par);
                        if (it == ov_prow.end()) { err = "rasilu0: overlap parent missing"; return CHIDG_GPU_EINVAL; }
                        en.parent = it->second;
                    }
                    en.a_off = A->voff[k];
                    en.t_off = A->voff[kt];
                    en.nc = A->bsize(par);
                    en.blk = -1;
                    P.lo[oi.pr].push_back(en);
                }
                for (int32_t k : oi.upper_blk) {
                    const int par = A->ce[k];
                    auto it = ov_prow.find(par);
                    if (it == ov_prow.end()) { err = "rasilu0: overlap parent missing"; return CHIDG_GPU_EINVAL; }
                    IluEntry en;
                    en.parent = it->second;
                    en.a_off = A->voff[k];
                    en.nc = A->bsize(par);
                    en.blk = -1;
                    P.up[oi.pr].push_back(en);
                }
            }
    }
    P.n_ext = ov_cursor;
    return CHIDG_GPU_OK;
}

// Rows of a level are inverted in groups of alike blocks: a launch takes the
// cluster size and the panel warps of its largest one.
static int inv_class(int b) { return b <= 64 ? 0 : b <= 136 ? 1 : b <= 208 ? 2 : b <= 320 ? 3 : b <= GJ_MAX ? 4 : 5; }

// Which rows of a streamed sweep are one task, and where every row's partial
// sums go.  Forward: a vector per slice of every entry; backward: the same (one
// vector for a one-task row), then one per slice of inv(D).
static void stream_layout(IluProgram& P) {
    const int np = (int)P.prow_b.size();
    P.part_s = 1;
    P.max_row_task_cols = 0;
    P.no_lower = true;
    for (const auto& ents : P.lo) P.no_lower = P.no_lower && ents.empty();
    for (int fwd = 1; fwd >= 0; --fwd) {
        std::vector<uint8_t>& whole = fwd ? P.whole_f : P.whole_b;
        std::vector<int64_t>& base = fwd ? P.base_f : P.base_u;
        whole.assign(np, 0);
        base.assign(np, 0);
        if (!fwd) P.base_d.assign(np, 0);
        int64_t size = 0;
        for (int pr = 0; pr < np; ++pr) {
            const auto& ents = (fwd ? P.lo : P.up)[pr];
            const int b = P.prow_b[pr], ns = P.slices(b);
            int cols = 0;
            for (const auto& en : ents) cols += en.nc;
            base[pr] = size;
            if (b <= SW_ROW_B && cols <= SW_ROW_COLS) {
                whole[pr] = 1;
                P.max_row_task_cols = std::max(P.max_row_task_cols, std::max(cols, b));
                if (!fwd && !ents.empty()) size += b;
                continue;
            }
            size += (int64_t)b * ns * ents.size();
            if (!fwd) {
                P.base_d[pr] = size;
                size += (int64_t)b * ns;
            }
        }
        P.part_s = std::max(P.part_s, size);
    }
    // the task-split schedule leaves one vector an entry in the same scratch:
    // sized for both, so that a change of the schedule never moves it (captured
    // sequences hold its address)
    for (int fwd = 1; fwd >= 0; --fwd) {
        int64_t size = 0;
        for (int pr = 0; pr < np; ++pr) size += (int64_t)P.prow_b[pr] * (int64_t)(fwd ? P.lo : P.up)[pr].size();
        P.part_s = std::max(P.part_s, size);
    }
}

// Tasks in key order (those of one key as added): their numbers first, then, after
// place(), the tasks themselves, each written where it stays.
struct KeyedTasks {
    int first;                        // the smallest key
    std::vector<int64_t> at;          // tasks of a key; then where its next one goes
    std::unique_ptr<StreamTask[]> task;
    int64_t n = 0;
    explicit KeyedTasks(int smallest) : first(smallest) {}
    void count(int key, int64_t tasks) {
        const size_t k = (size_t)(key - first);
        if (at.size() <= k) at.resize(k + 1, 0);
        at[k] += tasks;
    }
    void place() {
        for (int64_t& a : at) {
            const int64_t here = a;
            a = n;
            n += here;
        }
        task.reset(new StreamTask[(size_t)n]);    // (not zeroed: every one is written)
    }
    StreamTask& next(int key) { return task[(size_t)at[(size_t)(key - first)]++]; }
};

// The tasks of a streamed sweep with their keys: a slice of an entry follows
// the level of the row it waits for (2 lev(parent)), a whole row and the slices
// of inv(D) come just before the tasks that wait for the row (2 lev(row) - 1).  A
// task waits only for rows all of whose tasks have smaller keys.  Keys are
// scaled so that other tasks fit between them.
//
// A task takes all slices of a block where the level has `many` blocks or more:
// two an SM (24^3 of order 2, forward and backward sweep with matvec rows: 1139
// and 2830 us; with four 1140 and 2938, with one 1164 and 2811, never 1430 and
// 3145; 12^3: 260 and 491, 250 and 495, 296 and 523, 250 and 495).
// With mv_key the matvec rows' tasks are among them, at these keys.
static void stream_tasks(const IluProgram& P, bool fwd, const std::vector<int>& lev, int scale, int many, KeyedTasks& keyed,
                         const std::vector<int>* mv_key = nullptr) {
    // blocks per level: inv(D) by the row's, entries by the parent's
    std::vector<int> dlev, elev;
    for (int pr = 0; pr < (int)P.prow_b.size(); ++pr) {
        auto add = [](std::vector<int>& v, int l, int n) {
            if ((int)v.size() <= l) v.resize(l + 1, 0);
            v[l] += n;
        };
        add(dlev, lev[pr], 1);
        for (const auto& en : (fwd ? P.lo : P.up)[pr]) add(elev, lev[en.parent], 1);
    }
    const int np = (int)P.prow_b.size();
    const std::vector<uint8_t>& whole = fwd ? P.whole_f : P.whole_b;
    std::vector<int> first(np + 1, 0);
    for (int pr = 0; pr < np; ++pr) first[pr + 1] = first[pr] + (int)(fwd ? P.lo : P.up)[pr].size();
    // slices of a block that a task takes, by the blocks of its level
    auto diag_step = [&](int pr, int b, int ns) { return dlev[lev[pr]] >= many && sweep_groups_slices(b, P.diagonal) ? ns : 1; };
    auto entry_step = [&](int parent, int ns) { return elev[lev[parent]] >= many ? ns : 1; };
    for (int pr = 0; pr < np; ++pr) {
        const auto& ents = (fwd ? P.lo : P.up)[pr];
        const int b = P.prow_b[pr], ns = P.slices(b);
        if (mv_key) keyed.count((*mv_key)[pr], 1);
        if (whole[pr]) {
            keyed.count(scale * (2 * lev[pr] - 1), 1);
            continue;
        }
        if (!fwd) keyed.count(scale * (2 * lev[pr] - 1), ns / diag_step(pr, b, ns));
        for (const auto& en : ents) keyed.count(scale * (2 * lev[en.parent]), ns / entry_step(en.parent, ns));
        if (fwd && ents.empty()) keyed.count(-scale, 1);
    }
    keyed.place();
    for (int32_t pr : fwd ? P.fwd_rows : P.bwd_rows) {
        const auto& ents = (fwd ? P.lo : P.up)[pr];
        const int b = P.prow_b[pr], ns = P.slices(b), ne = (int)ents.size();
        StreamTask t{};
        t.row = pr;
        t.b = b;
        t.zrow = P.z_off[pr];
        t.vrow = P.v_off[pr];
        t.q0 = first[pr];
        t.q1 = first[pr + 1];
        t.wait = -1;
        t.par = pr;
        t.pb = b;
        t.ns = ns;
        if (whole[pr]) {
            t.code = SW_ROW;
            for (const auto& en : ents) t.cols += en.nc;
            t.off = fwd ? (ne ? ents[0].l_off : 0) : P.dinv_off[pr];
            t.out = t.rbase = fwd ? 0 : P.base_u[pr];
            t.nall = ne ? 1 : 0;
            t.src = !fwd && P.lo[pr].empty();
            keyed.next(scale * (2 * lev[pr] - 1)) = t;
            continue;
        }
        const int dstep = diag_step(pr, b, ns);
        if (!fwd)
            for (int s = 0; s < ns; s += dstep) {
                StreamTask& u = keyed.next(scale * (2 * lev[pr] - 1));
                u = t;
                u.nc = b;
                u.s0 = s;
                u.nsl = dstep;
                const int c0 = b * s / ns;
                u.code = SW_DIAG;
                u.cols = b * (s + dstep) / ns - c0;
                u.off = P.dinv_off[pr] + (int64_t)c0 * b;
                u.out = P.base_d[pr] + (int64_t)s * b;
                u.rbase = P.base_d[pr];
                u.nall = ns;
                u.wait = ne ? ne * ns : -1;
                u.npart = ne * ns;
                // z_r = v_r in a row without lower entries
                u.src = P.lo[pr].empty();
                u.seg = (u.src ? t.vrow : t.zrow) + c0;
                u.pseg = P.base_u[pr] + c0;
            }
        for (int e = 0; e < ne; ++e) {
            const int step = entry_step(ents[e].parent, ns);
            for (int s = 0; s < ns; s += step) {
                StreamTask& u = keyed.next(scale * (2 * lev[ents[e].parent]));
                u = t;
                u.nc = ents[e].nc;
                u.s0 = s;
                u.nsl = step;
                const int q = ents[e].parent, nc = ents[e].nc, c0 = nc * s / ns, nq = (int)(fwd ? P.lo : P.up)[q].size();
                const int nsq = P.slices(nc);
                u.code = SW_ENTRY;
                u.cols = nc * (s + step) / ns - c0;
                u.off = (fwd ? ents[e].l_off : ents[e].a_off) + (int64_t)c0 * b;
                u.rbase = fwd ? P.base_f[pr] : P.base_u[pr];
                u.out = u.rbase + (int64_t)(e * ns + s) * b;
                u.nall = ne * ns;
                u.par = q;
                u.pb = nc;
                if (whole[q]) {
                    u.wait = 0;
                    u.src = 0;
                    u.seg = P.z_off[q] + c0;
                } else if (fwd) {
                    u.wait = nq ? nq * nsq : -1;
                    u.npart = nq * nsq;
                    u.src = 1;
                    u.seg = P.v_off[q] + c0;
                    u.pseg = P.base_f[q] + c0;
                } else {
                    u.wait = nsq;
                    u.npart = nsq;
                    u.src = 2;
                    u.pseg = P.base_d[q] + c0;
                }
            }
        }
        if (fwd && ne == 0) {
            // z_r = v_r for whoever reads it (the backward sweep): a slice of no columns
            StreamTask& u = keyed.next(-scale);
            u = t;
            u.code = SW_ENTRY;
            u.rbase = u.out = P.base_f[pr];
            u.nall = 1;
            u.nsl = 1;
        }
    }
    if (mv_key)
        for (int r = 0; r < np; ++r) {
            StreamTask& t = keyed.next((*mv_key)[r]);
            t = StreamTask{};
            t.row = r;
            t.code = SW_MATVEC;
            t.b = P.prow_b[r];
            t.rbase = P.base_u[r];
            t.nall = P.up[r].empty() ? 0 : P.whole_b[r] ? 1 : (int)P.up[r].size() * P.slices(t.b);
            t.wait = -1;
        }
}

// Levels, LD slots, GEMM tasks, device upload.
static int finalize_program(chidg_gpu_ctx* ctx, const chidg_gpu_matrix* A, IluProgram& P) {
    const int np = (int)P.prow_b.size();
    P.nprow = np;
    // forward / factor levels: programme rows are listed in the reference's
    // processing order, so every lower parent precedes its row
    std::vector<int> lf(np, 0), lb(np, 0);
    for (int pr = 0; pr < np; ++pr) {
        int l = 0;
        for (auto& en : P.lo[pr]) {
            if (en.parent >= pr) return fail(ctx, CHIDG_GPU_EINVAL, "ilu programme: lower parent after its row");
            l = std::max(l, lf[en.parent] + 1);
        }
        lf[pr] = l;
    }
    for (int pr = np - 1; pr >= 0; --pr) {
        int l = 0;
        for (auto& en : P.up[pr]) {
            if (en.parent <= pr) return fail(ctx, CHIDG_GPU_EINVAL, "ilu programme: upper parent before its row");
            l = std::max(l, lb[en.parent] + 1);
        }
        lb[pr] = l;
    }
    auto bucket = [&](const std::vector<int>& lev, std::vector<int32_t>& rows, std::vector<int>& ptr) {
        int nl = 0;
        for (int v : lev) nl = std::max(nl, v + 1);
        ptr.assign(nl + 1, 0);
        for (int v : lev) ptr[v + 1]++;
        for (int l = 0; l < nl; ++l) ptr[l + 1] += ptr[l];
        rows.assign(lev.size(), 0);
        std::vector<int> cur(ptr.begin(), ptr.end() - 1);
        for (int pr = 0; pr < (int)lev.size(); ++pr) rows[cur[lev[pr]]++] = pr;
    };
    bucket(lf, P.fwd_rows, P.fwd_ptr);
    bucket(lb, P.bwd_rows, P.bwd_ptr);
    P.lb = lb;
    P.bmv_uid = -1;
    // LD slots: per programme row [inv(D)][L_1][L_2]...
    P.dinv_off.assign(np, 0);
    int64_t ld = 0;
    for (int pr = 0; pr < np; ++pr) {
        const int b = P.prow_b[pr];
        P.dinv_off[pr] = ld;
        ld += (int64_t)b * b;
        for (auto& en : P.lo[pr]) { en.l_off = ld; ld += (int64_t)b * en.nc; }
    }
    P.ld_size = ld;
    // streamed sweeps: the tasks in key order
    stream_layout(P);
    for (int fwd = 1; fwd >= 0; --fwd) {
        KeyedTasks keyed(-1);
        stream_tasks(P, fwd != 0, fwd ? lf : lb, 1, 2 * ctx->nsm, keyed);
        int st0;
        if ((st0 = upload_items(ctx, fwd ? P.d_sf_task : P.d_sb_task, keyed.task.get(), (size_t)keyed.n))) return st0;
        (fwd ? P.ntask_sf : P.ntask_sb) = (int)keyed.n;
    }
    // flatten entry lists
    std::vector<int32_t> lo_ptr(np + 1, 0), up_ptr(np + 1, 0), lo_par, up_par, lo_nc, up_nc;
    std::vector<int64_t> lo_L, up_U;
    for (int pr = 0; pr < np; ++pr) {
        for (auto& en : P.lo[pr]) { lo_par.push_back(en.parent); lo_nc.push_back(en.nc); lo_L.push_back(en.l_off); }
        for (auto& en : P.up[pr]) { up_par.push_back(en.parent); up_nc.push_back(en.nc); up_U.push_back(en.a_off); }
        lo_ptr[pr + 1] = (int32_t)lo_par.size();
        up_ptr[pr + 1] = (int32_t)up_par.size();
    }
    P.max_lo_cols = 0;
    P.max_up_cols = 0;
    P.max_b = 0;
    for (int pr = 0; pr < np; ++pr) {
        int c = 0;
        for (auto& en : P.lo[pr]) c += en.nc;
        P.max_lo_cols = std::max(P.max_lo_cols, c);
        c = 0;
        for (auto& en : P.up[pr]) c += en.nc;
        P.max_up_cols = std::max(P.max_up_cols, c);
        P.max_b = std::max(P.max_b, P.prow_b[pr]);
    }
    // factorisation schedule per forward level.  Rows of a level are ordered
    // by block-size class (inv_class); products of blocks that the FP32 tensor-core kernels take
    // come first in each level.
    std::vector<GemmTask> ltasks, stasks;
    std::vector<GemmPair> lpairs, spairs;
    std::vector<int32_t> ltask_of;          // first L task of the row at each position of fwd_rows (small blocks)
    P.ltask_ptr.assign(P.fwd_ptr.size(), 0);
    P.stask_ptr.assign(P.fwd_ptr.size(), 0);
    P.ltask_small.assign(P.fwd_ptr.size(), 0);
    P.stask_small.assign(P.fwd_ptr.size(), 0);
    P.inv_seg.clear();
    P.inv_seg_ptr.assign(P.fwd_ptr.size(), 0);
    const int nlev = (int)P.fwd_ptr.size() - 1;
    for (int l = 0; l < nlev; ++l) {
        std::stable_sort(P.fwd_rows.begin() + P.fwd_ptr[l], P.fwd_rows.begin() + P.fwd_ptr[l + 1],
                         [&](int32_t a, int32_t b2) { return inv_class(P.prow_b[a]) < inv_class(P.prow_b[b2]); });
        for (int i = P.fwd_ptr[l]; i < P.fwd_ptr[l + 1];) {
            const int cls = inv_class(P.prow_b[P.fwd_rows[i]]);
            int j = i, bmax = 0;
            for (; j < P.fwd_ptr[l + 1] && inv_class(P.prow_b[P.fwd_rows[j]]) == cls; ++j)
                bmax = std::max(bmax, P.prow_b[P.fwd_rows[j]]);
            P.inv_seg.push_back({i, j - i, bmax});
            i = j;
        }
        P.inv_seg_ptr[l + 1] = (int)P.inv_seg.size();
        // pass 0: products of blocks of at most FACTOR32_SMALL rows (the FP32
        // factorisation takes them on the tensor cores), pass 1: larger ones
        for (int pass = 0; pass < 2; ++pass) {
            for (int i = P.fwd_ptr[l]; i < P.fwd_ptr[l + 1]; ++i) {
                const int pr = P.fwd_rows[i];
                const int b = P.prow_b[pr];
                if (pass == 0) ltask_of.push_back((int32_t)ltasks.size());
                for (auto& en : P.lo[pr]) {
                    // L = A_lower * inv(D_parent)      (precon_ILU0.f90:231)
                    const bool small = b <= FACTOR32_SMALL && en.nc <= FACTOR32_SMALL;
                    if (small != (pass == 0)) continue;
                    GemmTask t{};
                    t.c_off = en.l_off; t.cinit_off = -1; t.m = b; t.n = en.nc;
                    t.q_begin = (int32_t)lpairs.size();
                    lpairs.push_back(GemmPair{en.a_off, P.dinv_off[en.parent], en.nc, 0});
                    t.q_end = (int32_t)lpairs.size();
                    t.elem = P.prow_elem[pr];
                    ltasks.push_back(t);
                }
                // D = A_diag - sum L * A(parent, itranspose)   (:238-239);
                // assembled rows get their D from k_assemble_rows instead
                if (P.assembled) continue;
                bool small = b <= FACTOR32_SMALL;
                for (auto& en : P.lo[pr]) small = small && en.nc <= FACTOR32_SMALL;
                if (small != (pass == 0)) continue;
                GemmTask t{};
                t.c_off = P.dinv_off[pr]; t.cinit_off = P.diagA_off[pr]; t.m = b; t.n = b;
                t.q_begin = (int32_t)spairs.size();
                for (auto& en : P.lo[pr]) spairs.push_back(GemmPair{en.l_off, en.t_off, en.nc, 0});
                t.q_end = (int32_t)spairs.size();
                t.elem = P.prow_elem[pr];
                stasks.push_back(t);
            }
            if (pass == 0) {
                P.ltask_small[l + 1] = (int)ltasks.size() - P.ltask_ptr[l];
                P.stask_small[l + 1] = (int)stasks.size() - P.stask_ptr[l];
            }
        }
        P.ltask_ptr[l + 1] = (int)ltasks.size();
        P.stask_ptr[l + 1] = (int)stasks.size();
    }
    int st;
    if ((st = upload_array(ctx, P.d_prow_b, P.prow_b)) || (st = upload_array(ctx, P.d_prow_elem, P.prow_elem)) ||
        (st = upload_array(ctx, P.d_v_off, P.v_off)) || (st = upload_array(ctx, P.d_z_off, P.z_off)) ||
        (st = upload_array(ctx, P.d_dinv_off, P.dinv_off)) || (st = upload_array(ctx, P.d_lo_ptr, lo_ptr)) ||
        (st = upload_array(ctx, P.d_lo_L, lo_L)) || (st = upload_array(ctx, P.d_lo_par, lo_par)) ||
        (st = upload_array(ctx, P.d_lo_nc, lo_nc)) || (st = upload_array(ctx, P.d_up_ptr, up_ptr)) ||
        (st = upload_array(ctx, P.d_up_U, up_U)) || (st = upload_array(ctx, P.d_up_par, up_par)) ||
        (st = upload_array(ctx, P.d_up_nc, up_nc)) || (st = upload_array(ctx, P.d_fwd_rows, P.fwd_rows)) ||
        (st = upload_array(ctx, P.d_bwd_rows, P.bwd_rows)) || (st = upload_array(ctx, P.d_ltasks, ltasks)) ||
        (st = upload_array(ctx, P.d_lpairs, lpairs)) || (st = upload_array(ctx, P.d_stasks, stasks)) ||
        (st = upload_array(ctx, P.d_spairs, spairs)) || (st = upload_array(ctx, P.d_ltask_of, ltask_of)))
        return st;
    P.rows.prow_b = (const int32_t*)P.d_prow_b.ptr;
    P.rows.v_off = (const int64_t*)P.d_v_off.ptr;
    P.rows.z_off = (const int64_t*)P.d_z_off.ptr;
    P.rows.dinv_off = (const int64_t*)P.d_dinv_off.ptr;
    P.rows.lo_ptr = (const int32_t*)P.d_lo_ptr.ptr;
    P.rows.lo_L = (const int64_t*)P.d_lo_L.ptr;
    P.rows.lo_par = (const int32_t*)P.d_lo_par.ptr;
    P.rows.lo_nc = (const int32_t*)P.d_lo_nc.ptr;
    P.rows.up_ptr = (const int32_t*)P.d_up_ptr.ptr;
    P.rows.up_U = (const int64_t*)P.d_up_U.ptr;
    P.rows.up_par = (const int32_t*)P.d_up_par.ptr;
    P.rows.up_nc = (const int32_t*)P.d_up_nc.ptr;
    P.sweep_threads = launch_dim_for(SW_GCAP, P.prow_b);
    if (P.assembled &&
        ((st = upload_array(ctx, P.d_asm_ptr, P.asm_ptr)) || (st = upload_array(ctx, P.d_asm_src, P.asm_src)) ||
         (st = upload_array(ctx, P.d_asm_r0, P.asm_r0)) || (st = upload_array(ctx, P.d_asm_c0, P.asm_c0)) ||
         (st = upload_array(ctx, P.d_asm_nr, P.asm_nr)) || (st = upload_array(ctx, P.d_asm_nc, P.asm_nc))))
        return st;
    (void)A;
    return CHIDG_GPU_OK;
}

void chidg::release_program(IluProgram& P) {
    for (Buffer* b : {&P.d_prow_b, &P.d_prow_elem, &P.d_v_off, &P.d_z_off, &P.d_dinv_off, &P.d_lo_ptr, &P.d_lo_L,
                      &P.d_lo_par, &P.d_lo_nc, &P.d_up_ptr, &P.d_up_U, &P.d_up_par, &P.d_up_nc, &P.d_fwd_rows,
                      &P.d_bwd_rows, &P.d_ltasks, &P.d_lpairs, &P.d_stasks, &P.d_spairs, &P.d_ltask_of, &P.d_tf_row, &P.d_tf_ent,
                      &P.d_tb_row, &P.d_tb_ent, &P.d_poff_f, &P.d_poff_b, &P.d_sf_task, &P.d_sb_task, &P.d_asm_ptr,
                      &P.d_asm_src, &P.d_asm_r0, &P.d_asm_c0, &P.d_asm_nr, &P.d_asm_nc, &P.d_bmv_task,
                      &P.d_col_prow, &P.d_mv_skip})
        release(*b);
    P.bmv_uid = -1;
}

// The ILU programme of M from A's pattern, or from A^T's when A->transposed
// (ILU0 and Jacobi of A^T, precon_ILU0.f90:148-207, precon_jacobi.f90:121-125).
// RASILU0 always uses A: the reference refuses transposed matrices there.
static int build_programme(chidg_gpu_precon* M, chidg_gpu_matrix* A) {
    chidg_gpu_ctx* ctx = M->ctx;
    chidg_gpu_matrix* S = A;
    int st;
    const bool own = M->kind == CHIDG_PRECON_RASILU0 || M->kind == CHIDG_PRECON_HB;   // built from A itself
    if (!own && (st = matrix_op(A, &S))) return st;
    std::string err;
    st = (M->kind == CHIDG_PRECON_RASILU0) ? build_rasilu0(S, M->P, err)
         : (M->kind == CHIDG_PRECON_HB)    ? build_hb(S, M->P, err)
                                           : build_ilu0(S, M->kind == CHIDG_PRECON_JACOBI, M->P, err);
    if (st) { release_program(M->P); return fail(ctx, st, err); }
    if ((st = finalize_program(ctx, S, M->P))) { release_program(M->P); return st; }
    const size_t sync_bytes = sizeof(unsigned) * (2 + 5 * (size_t)M->P.nprow);
    if ((st = ensure(ctx, M->sync, sync_bytes))) { release_program(M->P); return st; }
    cudaMemsetAsync(M->sync.ptr, 0, sync_bytes, ctx->stream);
    M->built_transposed = A->transposed && !own;
    return CHIDG_GPU_OK;
}

// The matrix whose blocks M factors and applies: A, or A^T for ILU0 / Jacobi
// of a transposed A.  RASILU0 with a transposed A is an error, as in the
// reference ("transpose not implemented for 'native' containers",
// precon_RASILU0.f90:254,494).
// precon_HB reads A's own blocks whether or not A is transposed, as the
// reference does (precon_HB.f90:169-310 does not consult A%transposed).
static int precon_source(chidg_gpu_precon* M, chidg_gpu_matrix** S) {
    chidg_gpu_matrix* A = M->A;
    if (A->transposed && M->kind == CHIDG_PRECON_RASILU0)
        return fail(M->ctx, CHIDG_GPU_EINVAL, "RASILU0: transpose not implemented for 'native' containers");
    if (M->kind == CHIDG_PRECON_HB) { *S = A; return CHIDG_GPU_OK; }
    return matrix_op(A, S);
}

extern "C" int chidg_gpu_precon_create(chidg_gpu_matrix* A, int32_t kind, chidg_gpu_precon** out) {
    if (!A || !out) return CHIDG_GPU_EINVAL;
    *out = nullptr;
    chidg_gpu_ctx* ctx = A->ctx;
    cudaSetDevice(ctx->device);
    if (kind < CHIDG_PRECON_IDENTITY || kind > CHIDG_PRECON_HB) return fail(ctx, CHIDG_GPU_EINVAL, "precon_create: unknown kind");
    auto* M = new chidg_gpu_precon();
    static std::atomic<int64_t> next_uid{1};
    M->uid = next_uid++;
    M->ctx = ctx;
    M->A = A;
    M->kind = kind;
    if (kind != CHIDG_PRECON_IDENTITY) {
        const int st = build_programme(M, A);
        if (st) { release(M->sync); delete M; return st; }
    }
    *out = M;
    return CHIDG_GPU_OK;
}

extern "C" int chidg_gpu_precon_destroy(chidg_gpu_precon* M) {
    if (!M) return CHIDG_GPU_OK;
    cudaSetDevice(M->ctx->device);
    cudaStreamSynchronize(M->ctx->stream);
    release_program(M->P);
    for (Buffer* b : {&M->LD, &M->LD32, &M->LD16, &M->zx, &M->zx32, &M->piv_scratch, &M->sync, &M->part64, &M->part32}) release(*b);
    delete M;
    return CHIDG_GPU_OK;
}
extern "C" int chidg_gpu_precon_stamp(chidg_gpu_precon* M, int64_t* s) {
    if (!M || !s) return CHIDG_GPU_EINVAL;
    *s = M->stamp;
    return CHIDG_GPU_OK;
}

// Whether `count` blocks of up to bmax rows are inverted sooner by one CTA a
// block (k_block_inverse_rows, one CTA an SM) than by clusters of C CTAs
// (k_block_inverse_gj).  Alone a block takes 2.6 (216 rows) to 3.7 times (352) as
// long in the first form, but 148 blocks run at a time in it, and some 50, 35 or
// 26 clusters of three, four or five.  bmax / 75 lies between the ratios measured
// at 216 to 352 rows and 30 to 740 blocks; where it chooses the first form that
// was never slower by more than 2 %, and the other choice cost up to 10 % at two
// waves of it.  ms of an update of one level, clusters / one CTA a block: 240 rows,
// 100 blocks 0.60 / 0.61, 148 0.80 / 0.65, 740 3.30 / 3.02; 270 rows, 60 blocks
// 0.49 / 0.76, 100 0.95 / 0.78, 740 5.38 / 3.89; 320 rows, 100 blocks 1.18 / 1.10,
// 148 1.75 / 1.21, 200 2.32 / 2.23, 740 8.30 / 5.90.  Up to 208 rows clusters of
// two always win (148 blocks 0.38 / 0.50).
template <typename K>
static bool rows_inverse_wins(chidg_gpu_ctx* ctx, K kern, const cudaLaunchConfig_t& cfg, int C, int count, int bmax) {
    if (bmax <= 208 || bmax > RP_MAX) return false;
    int& slots = ctx->gj_slots[C];
    if (slots == 0 && (cudaOccupancyMaxActiveClusters(&slots, kern, &cfg) != cudaSuccess || slots < 1)) {
        cudaGetLastError();
        slots = 1;
    }
    const long long waves = (count + slots - 1) / slots, rows_waves = (count + ctx->nsm - 1) / ctx->nsm;
    return 75 * waves > bmax * rows_waves;
}

// the inverses of rows row_begin .. + count of the factorisation order, blocks of at most bmax rows
static int launch_inverse(chidg_gpu_precon* M, int row_begin, int count, int bmax) {
    chidg_gpu_ctx* ctx = M->ctx;
    IluProgram& P = M->P;
    double* LD = (double*)M->LD.ptr;
    const int64_t* off = (const int64_t*)P.d_dinv_off.ptr;
    const int32_t *pb = (const int32_t*)P.d_prow_b.ptr, *pe = (const int32_t*)P.d_prow_elem.ptr,
                  *rows = (const int32_t*)P.d_fwd_rows.ptr;
    int st;
    if (bmax <= GJ_MAX) {
        const int C = gj_cluster(bmax), T = (gj_rows(bmax) + 31) / 32;
        // update warps (and, in a cluster, the one that pushes the panels): the
        // products take about as long as the panel with two tiles a warp
        const int threads = 32 * std::min(GJ_THREADS / 32, T + (bmax <= 64 ? 2 : 7));
        const size_t smem = gj_smem(bmax, C);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(count * C));
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = ctx->stream;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)C;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = C > 1 ? 1 : 0;
        auto go = [&](auto kern) -> int {
            const int s2 = raise_smem_limit((const void*)kern, smem);
            if (s2) return fail(ctx, s2, "block inverse shared memory");
            if (rows_inverse_wins(ctx, kern, cfg, C, count, bmax)) return 1;
            const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, LD, off, pb, pe, rows, row_begin, ctx->d_status, C, T);
            if (e != cudaSuccess) {
                cudaGetLastError();
                return cuda_fail(ctx, e, "k_block_inverse_gj");
            }
            return check_launch(ctx, "k_block_inverse_gj");
        };
        if (C == 1) return T <= 4 ? go(k_block_inverse_gj<false, 4>) : go(k_block_inverse_gj<false, 8>);
        st = T <= 8 ? go(k_block_inverse_gj<true, 8>) : go(k_block_inverse_gj<true, 12>);
        if (st != 1) return st;
        const size_t rsmem = rp_smem_bytes(bmax);
        if ((st = raise_smem_limit((const void*)k_block_inverse_rows, rsmem)))
            return fail(ctx, st, "row inverse shared memory");
        k_block_inverse_rows<<<count, RP_THREADS, rsmem, ctx->stream>>>(LD, off, pb, pe, rows, row_begin, ctx->d_status, bmax);
        return check_launch(ctx, "k_block_inverse_rows");
    }
    // larger blocks: panels of 16 columns (8 above 704 rows) in shared memory,
    // (2 NB + 1) b doubles
    if ((st = ensure(ctx, M->piv_scratch, sizeof(int) * 1024 * (size_t)std::max(count, 1)))) return st;
    auto go = [&](auto kern, int nbw) -> int {
        const size_t smem = sizeof(double) * (size_t)(2 * nbw + 1) * bmax;
        const int s2 = raise_smem_limit((const void*)kern, smem);
        if (s2) return fail(ctx, s2, "panel inverse shared memory");
        kern<<<count, 256, smem, ctx->stream>>>(LD, off, pb, pe, rows, row_begin, ctx->d_status, (int*)M->piv_scratch.ptr);
        return CHIDG_GPU_OK;
    };
    if ((st = bmax <= 704 ? go(k_block_inverse_panels<16>, 16) : go(k_block_inverse_panels<8>, 8))) return st;
    return check_launch(ctx, "k_block_inverse_panels");
}

// precon%update for the mixed-precision inner solves (MIXED_FP32, MIXED_BF16):
// the L and S products in FP32 (from the FP32 copy of A), the diagonal
// inverses in FP64 (the products' D blocks are written in FP64, inverted as in the
// FP64 factorisation and copied to FP32 per wavefront).  Only the FP32 (and
// BF16) factors are produced; LD's FP64 L blocks are not.
// The products of blocks up to 136 rows run on the tcgen05 tensor cores
// (k_task_gemm_umma), larger ones on the SIMT tiled kernel, which the FP64
// products' tensor-core tiles have overtaken: batched solves of orders 1 to 3 with
// FP32 inner solves run at 0.90 of the FP64 ones.  CHIDG_FACTOR32_MMA=sync selects
// the mma.sync TF32 kernel and CHIDG_FACTOR32_SIMT=1 the FP32 SIMT products
// (comparison runs)
static int factor32_kernel_env() {       // 0 tcgen05, 1 mma.sync, 2 SIMT
    static const int v = [] {
        const char* s = std::getenv("CHIDG_FACTOR32_SIMT");
        if (s && s[0] == '1') return 2;
        const char* m = std::getenv("CHIDG_FACTOR32_MMA");
        return (m && std::strcmp(m, "sync") == 0) ? 1 : 0;
    }();
    return v;
}

static int factor_fp32(chidg_gpu_precon* M, chidg_gpu_matrix* A, int precision) {
    chidg_gpu_ctx* ctx = M->ctx;
    IluProgram& P = M->P;
    int st;
    if ((st = matrix_lowp(A, CHIDG_GPU_MIXED_FP32))) return st;
    if (precision == CHIDG_GPU_MIXED_BF16 && (st = matrix_lowp(A, CHIDG_GPU_MIXED_BF16))) return st;
    if ((st = ensure(ctx, M->LD, sizeof(double) * (size_t)P.ld_size)) ||
        (st = ensure(ctx, M->LD32, sizeof(float) * (size_t)P.ld_size)))
        return st;
    const int kern = factor32_kernel_env();
    if ((st = raise_smem_limit((const void*)k_task_gemm_f32<float>, SF_SMEM)) ||
        (st = raise_smem_limit((const void*)k_task_gemm_f32<double>, SF_SMEM)) ||
        (st = raise_smem_limit((const void*)k_task_gemm_tf32<float>, ST_SMEM)) ||
        (st = raise_smem_limit((const void*)k_task_gemm_tf32<double>, ST_SMEM)) ||
        (st = raise_smem_limit((const void*)k_task_gemm_umma<float>, UM_SMEM)) ||
        (st = raise_smem_limit((const void*)k_task_gemm_umma<double>, UM_SMEM)))
        return fail(ctx, st, "FP32 factor GEMM shared memory");
    int* wstat = (int*)(ctx->d_scal + kSlotStatus);
    cudaMemsetAsync(ctx->d_scal + kSlotStatus, 0, sizeof(double), ctx->stream);
    const int nlev = (int)P.fwd_ptr.size() - 1;
    const float* A32 = (const float*)A->val32.ptr;
    float* L32 = (float*)M->LD32.ptr;
    double* LD = (double*)M->LD.ptr;
    const int ph = prof_begin(ctx, kProfFactor);
    // products of blocks above 136 rows (the tasks after the first
    // ltask_small / stask_small of a level): the SIMT tiled kernel in FP32
    const int tiles_1d = (P.max_b + GT_M - 1) / GT_M;
    for (int l = 0; l < nlev; ++l) {
        const int pg = prof_begin(ctx, kProfFactorGemm);
        const int nl_all = P.ltask_ptr[l + 1] - P.ltask_ptr[l], nl = P.ltask_small[l + 1];
        const int ns_all = P.stask_ptr[l + 1] - P.stask_ptr[l];
        const GemmTask* lt = (const GemmTask*)P.d_ltasks.ptr + P.ltask_ptr[l];
        const GemmTask* stt = (const GemmTask*)P.d_stasks.ptr + P.stask_ptr[l];
        if (nl_all > nl) {
            k_task_gemm<float, float, float, float><<<(nl_all - nl) * tiles_1d * tiles_1d, 256, 0, ctx->stream>>>(
                lt + nl, (const GemmPair*)P.d_lpairs.ptr, tiles_1d, tiles_1d, A32, L32, nullptr, L32, 1.0);
            if ((st = check_launch(ctx, "factor L products (FP32, large blocks)"))) return st;
        }
        if (nl > 0) {
            if (kern == 2)
                k_task_gemm_f32<float><<<nl, 256, SF_SMEM, ctx->stream>>>(lt, (const GemmPair*)P.d_lpairs.ptr, A32, L32,
                                                                         nullptr, L32, 1.0);
            else if (kern == 1)
                k_task_gemm_tf32<float><<<nl, ST_THREADS, ST_SMEM, ctx->stream>>>(lt, (const GemmPair*)P.d_lpairs.ptr, A32,
                                                                                 L32, nullptr, L32, 1.0);
            else
                k_task_gemm_umma<float><<<std::min(2 * nl, 2 * ctx->nsm), UM_THREADS, UM_SMEM, ctx->stream>>>(
                    lt, 2 * nl, (const GemmPair*)P.d_lpairs.ptr, A32, L32, nullptr, L32, 1.0, wstat, kSpinLimit);
            if ((st = check_launch(ctx, "factor L products (FP32 / TF32)"))) return st;
        }
        const int ns = P.stask_small[l + 1];
        if (ns_all > ns) {
            k_task_gemm<float, float, double, float><<<(ns_all - ns) * tiles_1d * tiles_1d, 256, 0, ctx->stream>>>(
                stt + ns, (const GemmPair*)P.d_spairs.ptr, tiles_1d, tiles_1d, L32, A32, (const double*)A->val.ptr, LD, -1.0);
            if ((st = check_launch(ctx, "factor S products (FP32, large blocks)"))) return st;
        }
        if (ns > 0) {
            if (kern == 2)
                k_task_gemm_f32<double><<<ns, 256, SF_SMEM, ctx->stream>>>(stt, (const GemmPair*)P.d_spairs.ptr, L32, A32,
                                                                          (const double*)A->val.ptr, LD, -1.0);
            else if (kern == 1)
                k_task_gemm_tf32<double><<<ns, ST_THREADS, ST_SMEM, ctx->stream>>>(stt, (const GemmPair*)P.d_spairs.ptr, L32,
                                                                                  A32, (const double*)A->val.ptr, LD, -1.0);
            else
                k_task_gemm_umma<double><<<std::min(2 * ns, 2 * ctx->nsm), UM_THREADS, UM_SMEM, ctx->stream>>>(
                    stt, 2 * ns, (const GemmPair*)P.d_spairs.ptr, L32, A32, (const double*)A->val.ptr, LD, -1.0, wstat,
                    kSpinLimit);
            if ((st = check_launch(ctx, "factor S products (FP32 / TF32)"))) return st;
        }
        prof_end(ctx, pg);
        const int pi = prof_begin(ctx, kProfFactorInv);
        for (int q = P.inv_seg_ptr[l]; q < P.inv_seg_ptr[l + 1]; ++q)
            if ((st = launch_inverse(M, P.inv_seg[q][0], P.inv_seg[q][1], P.inv_seg[q][2]))) return st;
        const int cnt = P.fwd_ptr[l + 1] - P.fwd_ptr[l];
        if (cnt > 0) {
            k_convert_dinv<<<cnt, 256, 0, ctx->stream>>>(LD, L32, (const int64_t*)P.d_dinv_off.ptr,
                                                         (const int32_t*)P.d_prow_b.ptr, (const int32_t*)P.d_fwd_rows.ptr,
                                                         P.fwd_ptr[l]);
            if ((st = check_launch(ctx, "k_convert_dinv"))) return st;
        }
        prof_end(ctx, pi);
    }
    prof_end(ctx, ph);
    if (precision == CHIDG_GPU_MIXED_BF16) {
        if ((st = ensure(ctx, M->LD16, sizeof(__nv_bfloat16) * (size_t)P.ld_size))) return st;
        k_convert<float, __nv_bfloat16><<<grid_for(P.ld_size, 256, ctx->nsm * 8), 256, 0, ctx->stream>>>(
            P.ld_size, (const float*)M->LD32.ptr, (__nv_bfloat16*)M->LD16.ptr);
        if ((st = check_launch(ctx, "k_convert LD32->LD16"))) return st;
    }
    return CHIDG_GPU_OK;
}

// precon%update: FP64 factorisation level by level, then the low-precision
// copies of the factors when requested.
extern "C" int chidg_gpu_precon_update(chidg_gpu_precon* M, chidg_gpu_matrix* A, int32_t precision) {
    if (!M || !A || A != M->A) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = M->ctx;
    cudaSetDevice(ctx->device);
    if (precision < CHIDG_GPU_FP64 || precision > CHIDG_GPU_MIXED_PRECON_FP32) return fail(ctx, CHIDG_GPU_EINVAL, "precon_update: bad precision");
    ctx->err_elem = -1;
    if (M->kind == CHIDG_PRECON_IDENTITY) { M->stamp = A->stamp; M->precision = precision; return CHIDG_GPU_OK; }
    int st;
    chidg_gpu_matrix* user = A;
    if ((st = precon_source(M, &A))) return st;          // from here on A is the matrix factored (A or A^T)
    if (M->kind != CHIDG_PRECON_RASILU0 && M->kind != CHIDG_PRECON_HB && M->built_transposed != user->transposed) {
        // the transposed flag changed since the programme was built
        cudaStreamSynchronize(ctx->stream);
        release_program(M->P);
        M->stamp = 0;
        if ((st = build_programme(M, user))) return st;
    }
    IluProgram& P = M->P;
    if ((st = ensure(ctx, M->LD, sizeof(double) * (size_t)P.ld_size))) return st;
    int big = INT_MAX;
    cudaMemcpyAsync(ctx->d_status, &big, sizeof(int), cudaMemcpyHostToDevice, ctx->stream);
    // fresh task counters for the task-split sweeps (a sweep cut short by an
    // error would otherwise leave them out of step)
    if (M->sync.ptr)
        cudaMemsetAsync((unsigned*)M->sync.ptr + 2 + P.nprow, 0, sizeof(unsigned) * 4 * (size_t)P.nprow, ctx->stream);
    if ((precision == CHIDG_GPU_MIXED_FP32 || precision == CHIDG_GPU_MIXED_BF16) && !P.assembled) {
        // the inner solves only read FP32 / BF16 factors: compute them in FP32
        if ((st = factor_fp32(M, A, precision))) return st;
        cudaMemcpyAsync(ctx->h_status, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
        const cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "precon update");
        double w = 0.0;
        if ((st = fetch_scalars(ctx, kSlotStatus, 1, &w))) return st;
        int wi = 0;
        std::memcpy(&wi, &w, sizeof(int));
        if (wi != 0) return fail(ctx, CHIDG_GPU_ETIMEOUT, "factor: a bounded wait for the tensor cores ran out");
        if (ctx->h_status[0] != INT_MAX) {
            ctx->err_elem = ctx->h_status[0];
            return fail(ctx, CHIDG_GPU_ESINGULAR, "inv: Matrix is numerically singular! (element " + std::to_string(ctx->h_status[0]) + ")");
        }
        M->ld64_valid = false;
        M->precision = precision;
        M->stamp = user->stamp;
        return CHIDG_GPU_OK;
    }
    const int nlev = (int)P.fwd_ptr.size() - 1;
    // CTA tiles per side of the largest output (k_task_gemm_f64)
    const int parts = fg_parts(P.max_b);
    if ((st = raise_smem_limit((const void*)k_task_gemm_f64, FG_SMEM))) return fail(ctx, st, "factor GEMM shared memory");
    const int ph = prof_begin(ctx, kProfFactor);
    if (P.assembled) {
        k_assemble_rows<<<P.nprow, 256, 0, ctx->stream>>>((double*)M->LD.ptr, (const int64_t*)P.d_dinv_off.ptr,
                                                         (const int32_t*)P.d_prow_b.ptr, (const double*)A->val.ptr,
                                                         (const int32_t*)P.d_asm_ptr.ptr, (const int64_t*)P.d_asm_src.ptr,
                                                         (const int32_t*)P.d_asm_r0.ptr, (const int32_t*)P.d_asm_c0.ptr,
                                                         (const int32_t*)P.d_asm_nr.ptr, (const int32_t*)P.d_asm_nc.ptr);
        if ((st = check_launch(ctx, "k_assemble_rows"))) return st;
    }
    // one launch for programmes of small blocks, else three a wavefront
    const bool by_rows = P.max_b <= FR_MAX && !P.assembled;
    if (by_rows) {
        const size_t smem = fr_smem(P.max_b);
        if ((st = raise_smem_limit((const void*)k_factor_rows, smem))) return fail(ctx, st, "factor rows shared memory");
        const int per_sm = resident_ctas((const void*)k_factor_rows, FG_THREADS, smem);
        if (per_sm < 1) return fail(ctx, CHIDG_GPU_EINVAL, "factor rows: does not fit an SM");
        unsigned* sync = (unsigned*)M->sync.ptr;
        cudaMemsetAsync(sync, 0, sizeof(unsigned), ctx->stream);
        cudaMemsetAsync(ctx->d_scal + kSlotStatus, 0, sizeof(double), ctx->stream);
        const FactorRows FR{(const GemmTask*)P.d_ltasks.ptr, (const GemmTask*)P.d_stasks.ptr, (const GemmPair*)P.d_lpairs.ptr,
                            (const GemmPair*)P.d_spairs.ptr, (const int32_t*)P.d_fwd_rows.ptr, P.rows.prow_b,
                            (const int32_t*)P.d_prow_elem.ptr, P.rows.lo_ptr, P.rows.lo_par, (const int32_t*)P.d_ltask_of.ptr,
                            P.rows.dinv_off, P.nprow};
        SweepSync S{sync, sync + 2, ++M->epoch, (int*)(ctx->d_scal + kSlotStatus), kSpinLimit};
        k_factor_rows<<<std::min(P.nprow, per_sm * ctx->nsm), FG_THREADS, smem, ctx->stream>>>(
            FR, (const double*)A->val.ptr, (double*)M->LD.ptr, S, ctx->d_status);
        if ((st = check_launch(ctx, "k_factor_rows"))) return st;
    }
    for (int l = 0; l < nlev && !by_rows; ++l) {
        const int pg = prof_begin(ctx, kProfFactorGemm);
        const int nl = P.ltask_ptr[l + 1] - P.ltask_ptr[l], ns = P.stask_ptr[l + 1] - P.stask_ptr[l];
        if (nl > 0) {
            k_task_gemm_f64<<<nl * parts * parts, FG_THREADS, FG_SMEM, ctx->stream>>>(
                (const GemmTask*)P.d_ltasks.ptr + P.ltask_ptr[l], (const GemmPair*)P.d_lpairs.ptr, parts, parts,
                (const double*)A->val.ptr, (const double*)M->LD.ptr, nullptr, (double*)M->LD.ptr, 1.0);
            if ((st = check_launch(ctx, "k_task_gemm_f64 L"))) return st;
        }
        if (ns > 0) {
            k_task_gemm_f64<<<ns * parts * parts, FG_THREADS, FG_SMEM, ctx->stream>>>(
                (const GemmTask*)P.d_stasks.ptr + P.stask_ptr[l], (const GemmPair*)P.d_spairs.ptr, parts, parts,
                (const double*)M->LD.ptr, (const double*)A->val.ptr, (const double*)A->val.ptr, (double*)M->LD.ptr, -1.0);
            if ((st = check_launch(ctx, "k_task_gemm_f64 S"))) return st;
        }
        prof_end(ctx, pg);
        const int pi = prof_begin(ctx, kProfFactorInv);
        for (int q = P.inv_seg_ptr[l]; q < P.inv_seg_ptr[l + 1]; ++q)
            if ((st = launch_inverse(M, P.inv_seg[q][0], P.inv_seg[q][1], P.inv_seg[q][2]))) return st;
        prof_end(ctx, pi);
    }
    prof_end(ctx, ph);
    cudaMemcpyAsync(ctx->h_status, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (by_rows) {
        double w = 0.0;
        if ((st = fetch_scalars(ctx, kSlotStatus, 1, &w))) return st;
        if ((st = status_word(ctx, w))) return st;
    }
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "precon update");
    if (ctx->h_status[0] != INT_MAX) {
        ctx->err_elem = ctx->h_status[0];
        return fail(ctx, CHIDG_GPU_ESINGULAR, "inv: Matrix is numerically singular! (element " + std::to_string(ctx->h_status[0]) + ")");
    }
    if (precision != CHIDG_GPU_FP64) {
        if ((st = matrix_lowp(A, precision))) return st;
        if (precision == CHIDG_GPU_MIXED_FP32 || precision == CHIDG_GPU_MIXED_PRECON_FP32) {
            if ((st = ensure(ctx, M->LD32, sizeof(float) * (size_t)P.ld_size))) return st;
            k_convert<double, float><<<grid_for(P.ld_size, 256, ctx->nsm * 8), 256, 0, ctx->stream>>>(P.ld_size, (const double*)M->LD.ptr, (float*)M->LD32.ptr);
        } else {
            if ((st = ensure(ctx, M->LD16, sizeof(__nv_bfloat16) * (size_t)P.ld_size))) return st;
            k_convert<double, __nv_bfloat16><<<grid_for(P.ld_size, 256, ctx->nsm * 8), 256, 0, ctx->stream>>>(P.ld_size, (const double*)M->LD.ptr, (__nv_bfloat16*)M->LD16.ptr);
        }
        if ((st = check_launch(ctx, "k_convert LD"))) return st;
    }
    M->ld64_valid = true;
    M->precision = precision;
    M->stamp = user->stamp;
    return CHIDG_GPU_OK;
}

// z = M^{-1} v in the given arithmetic.  TV is the vector type; factors come
// from LD (FP64), LD32 or LD16 by precision; U blocks from A (FP64 or FP32).
// Both sweeps as two dependency-driven launches (CHIDG_SCHED_DATAFLOW).
template <typename TL, typename TU, typename TV>
static int dataflow_sweeps(chidg_gpu_precon* M, const TL* LD, const TU* U, const TV* v, TV* zx, int variant) {
    chidg_gpu_ctx* ctx = M->ctx;
    IluProgram& P = M->P;
    using ACC = typename AccOf<TV>::type;
    const int threads = P.sweep_threads;
    const size_t smem = sizeof(ACC) * ((size_t)std::max(P.max_lo_cols, P.max_up_cols) + P.max_b + threads) + 512;
    auto kf = k_ilu_sweep_sf<TL, TU, TV, ACC, true>;
    auto kb = k_ilu_sweep_sf<TL, TU, TV, ACC, false>;
    int st;
    if ((st = raise_smem_limit((const void*)kf, smem)) || (st = raise_smem_limit((const void*)kb, smem)))
        return fail(ctx, st, "dataflow sweep shared memory");
    if (M->sf_grid[variant] == 0) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kb, threads, smem) != cudaSuccess || per_sm < 1) {
            cudaGetLastError();
            per_sm = 1;
        }
        M->sf_grid[variant] = std::max(1, std::min(P.nprow, per_sm * ctx->nsm));
    }
    const int grid = M->sf_grid[variant];
    unsigned* counters = (unsigned*)M->sync.ptr;
    SweepSync S{counters, counters + 2, 0u, (int*)(ctx->d_scal + kSlotStatus), kSpinLimit};
    cudaError_t e = cudaMemsetAsync(counters, 0, sizeof(unsigned) * (2 + 5 * (size_t)P.nprow), ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "sweep counters");
    int ph = prof_begin(ctx, sizeof(TV) == 8 ? kProfIluForward : kProfIlu32);
    S.epoch = ++M->epoch;
    S.counter = counters;
    kf<<<grid, threads, smem, ctx->stream>>>(P.rows, LD, U, (const int32_t*)P.d_fwd_rows.ptr, P.nprow, v, zx, S);
    if ((st = check_launch(ctx, "k_ilu_sweep_sf forward"))) return st;
    if (sizeof(TV) == 8) {
        prof_end(ctx, ph);
        ph = prof_begin(ctx, kProfIluBackward);
    }
    S.epoch = ++M->epoch;
    S.counter = counters + 1;
    kb<<<grid, threads, smem, ctx->stream>>>(P.rows, LD, U, (const int32_t*)P.d_bwd_rows.ptr, P.nprow, v, zx, S);
    if ((st = check_launch(ctx, "k_ilu_sweep_sf backward"))) return st;
    prof_end(ctx, ph);
    return CHIDG_GPU_OK;
}

// The task-split sweeps' lists, built when that schedule first runs: one task per
// entry, combine-only tasks for rows without entries; hand-out order by the
// level of the parent row.
static int build_split_tasks(chidg_gpu_ctx* ctx, IluProgram& P) {
    if (P.d_tf_row.ptr != nullptr) return CHIDG_GPU_OK;
    const int np = P.nprow;
    std::vector<int> lf(np, 0);
    for (int l = 0; l + 1 < (int)P.fwd_ptr.size(); ++l)
        for (int i = P.fwd_ptr[l]; i < P.fwd_ptr[l + 1]; ++i) lf[P.fwd_rows[i]] = l;
    for (int fwd = 0; fwd < 2; ++fwd) {
        const std::vector<int>& lev = fwd ? lf : P.lb;
        std::vector<std::pair<int, std::pair<int32_t, int32_t>>> keyed;
        std::vector<int> first(np + 1, 0);
        for (int pr = 0; pr < np; ++pr) first[pr + 1] = first[pr] + (int)(fwd ? P.lo : P.up)[pr].size();
        std::vector<int64_t> poff(first[np]);
        int64_t psize = 0;
        for (int pr = 0; pr < np; ++pr)
            for (int e = first[pr]; e < first[pr + 1]; ++e) { poff[e] = psize; psize += P.prow_b[pr]; }
        for (int32_t pr : fwd ? P.fwd_rows : P.bwd_rows) {
            const auto& ents = (fwd ? P.lo : P.up)[pr];
            if (ents.empty()) keyed.push_back({-1, {pr, -1}});
            for (size_t e = 0; e < ents.size(); ++e) keyed.push_back({lev[ents[e].parent], {pr, first[pr] + (int32_t)e}});
        }
        std::stable_sort(keyed.begin(), keyed.end(), [](const auto& a, const auto& c) { return a.first < c.first; });
        std::vector<int32_t> row, ent;
        for (auto& k : keyed) { row.push_back(k.second.first); ent.push_back(k.second.second); }
        (fwd ? P.ntask_f : P.ntask_b) = (int)row.size();
        int st;
        // (the forward rows last: they say that the lists are there)
        if ((st = upload_array(ctx, fwd ? P.d_poff_f : P.d_poff_b, poff)) ||
            (st = upload_array(ctx, fwd ? P.d_tf_ent : P.d_tb_ent, ent)) ||
            (st = upload_array(ctx, fwd ? P.d_tf_row : P.d_tb_row, row)))
            return st;
    }
    return CHIDG_GPU_OK;
}

// Both sweeps as two task-split launches (CHIDG_SCHED_TASKS).
template <typename TL, typename TU, typename TV>
static int task_sweeps(chidg_gpu_precon* M, const TL* LD, const TU* U, const TV* v, TV* zx, int variant) {
    chidg_gpu_ctx* ctx = M->ctx;
    IluProgram& P = M->P;
    using ACC = typename AccOf<TV>::type;
    // column-group budget of one task CTA; CHIDG_TASK_THREADS (a multiple of 32
    // up to 1024) narrows it for tuning
    static const int tk_cap_env = [] {
        const char* e = std::getenv("CHIDG_TASK_THREADS");
        const int v = e ? std::atoi(e) : 0;
        return (v >= 32 && v <= 1024 && v % 32 == 0) ? v : TK_GCAP;
    }();
    const int gcap = tk_cap_env;
    const int threads = launch_dim_for(gcap, P.prow_b);
    const size_t smem = sizeof(ACC) * 3 * 1024 + 512;
    auto kf = k_ilu_tasks<TL, TU, TV, ACC, true>;
    auto kb = k_ilu_tasks<TL, TU, TV, ACC, false>;
    if (M->tk_grid[variant] == 0) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kb, threads, smem) != cudaSuccess || per_sm < 1) {
            cudaGetLastError();
            per_sm = 1;
        }
        M->tk_grid[variant] = std::max(1, per_sm * ctx->nsm);
    }
    Buffer& pb = (sizeof(ACC) == 8) ? M->part64 : M->part32;
    int st = ensure(ctx, pb, sizeof(ACC) * (size_t)P.part_s);
    if (st || (st = build_split_tasks(ctx, P))) return st;
    unsigned* sync = (unsigned*)M->sync.ptr;
    unsigned* flags = sync + 2;
    SweepSync S{sync, flags, 0u, (int*)(ctx->d_scal + kSlotStatus), kSpinLimit};
    cudaError_t e = cudaMemsetAsync(sync, 0, sizeof(unsigned) * (2 + 5 * (size_t)P.nprow), ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "sweep counters");
    int ph = prof_begin(ctx, sizeof(TV) == 8 ? kProfIluForward : kProfIlu32);
    S.epoch = ++M->epoch;
    S.counter = sync;
    SweepTasks Tf{(const int32_t*)P.d_tf_row.ptr, (const int32_t*)P.d_tf_ent.ptr, (const int64_t*)P.d_poff_f.ptr,
                  flags + P.nprow};
    kf<<<std::min(M->tk_grid[variant], P.ntask_f), threads, smem, ctx->stream>>>(P.rows, LD, U, Tf, P.ntask_f, v, zx, (ACC*)pb.ptr, S, gcap);
    if ((st = check_launch(ctx, "k_ilu_tasks forward"))) return st;
    if (sizeof(TV) == 8) {
        prof_end(ctx, ph);
        ph = prof_begin(ctx, kProfIluBackward);
    }
    S.epoch = ++M->epoch;
    S.counter = sync + 1;
    SweepTasks Tb{(const int32_t*)P.d_tb_row.ptr, (const int32_t*)P.d_tb_ent.ptr, (const int64_t*)P.d_poff_b.ptr,
                  flags + 2 * P.nprow};
    kb<<<std::min(M->tk_grid[variant], P.ntask_b), threads, smem, ctx->stream>>>(P.rows, LD, U, Tb, P.ntask_b, v, zx, (ACC*)pb.ptr, S, gcap);
    if ((st = check_launch(ctx, "k_ilu_tasks backward"))) return st;
    prof_end(ctx, ph);
    return CHIDG_GPU_OK;
}

// The shape table: per kernel kind, block-size class and value width.
// Defaults of the sweeps: 8 consumer warps and two stages (four where every row
// is one task of few bytes) of 24 KB forward and 26 KB backward, which slices fill
// evenly: 45 columns of 135 rows are three chunks of the one, so that four CTAs
// share an SM, and two of the other; 40 columns of 320 rows five and four.  The
// stage size is the same in every class, so that a row is chunked, and sums, the
// same whatever the largest block beside it.  Forward sweep and backward sweep
// with matvec rows within FP64 solves, us, 24 / 26 KB: 24^3 of order 2 1137 / 1207
// and 3229 / 2957, 12^3 250 / 240 and 555 / 496, 9 x 8 x 10 of order 3 346 / 362
// and 882 / 851; 20 KB 1160, 249, 357 and 2941, 527, 950.  25 KB forward (two chunks
// of 23 columns and four CTAs an SM) is faster at 135 rows, 1034 against 1124 us at
// 24^3 and 127 against 141 at 8^3, but not at 320 rows (9 x 8 x 10: 375 against
// 346); the autotuner finds it.
// Programmes without couplings (Jacobi, precon_HB) have no chain, only as many
// copies in flight as CTAs fit: their backward sweep takes two stages of 24 KB, four
// CTAs an SM, and with the matvec rows of blocks up to 64 rows 20 KB (24^3 elements
// of 40 rows, Jacobi: apply 125 us with the other defaults, 83 with these, with
// matvec rows 614 and 397; 990 blocks of 280 rows 147 and 131).
// CHIDG_STREAM_SHAPE="warps,stages,kbytes" overrides the sweeps' defaults
// (comparison runs).
namespace {
std::mutex g_shape_mu;
StreamShape g_shape[kShapeKinds][kShapeClasses][3], g_default[kShapeKinds][kShapeClasses][3];
bool g_shape_init = false;
int width_slot(int esz) { return esz >= 8 ? 0 : esz == 4 ? 1 : 2; }
void init_shapes() {
    StreamShape sweep;
    bool given = false;
    if (const char* e = std::getenv("CHIDG_STREAM_SHAPE")) {
        int cw = 0, ns = 0, kb = 0;
        if (std::sscanf(e, "%d,%d,%d", &cw, &ns, &kb) == 3 && (cw == 4 || cw == 8 || cw == 16) && ns >= 2 &&
            ns <= SS_MAX_STAGES && kb >= 2 && kb <= 96)
            { sweep = StreamShape{cw, ns, kb * 1024}; given = true; }
    }
    for (int c = 0; c < kShapeClasses; ++c)
        for (int w = 0; w < 3; ++w) {
            const StreamShape def{8, c == 0 ? 4 : 2, 26 * 1024, true};
            g_shape[kShapeForward][c][w] = given ? sweep : StreamShape{8, def.nstage, 24 * 1024, true};
            g_shape[kShapeBackward][c][w] = given ? sweep : def;
            g_shape[kShapeBackwardMv][c][w] = def;
            g_shape[kShapeMatvec][c][w] = StreamShape{8, 2, 24 * 1024, true};
            for (int k = 0; k < kShapeKinds; ++k) g_default[k][c][w] = g_shape[k][c][w];
        }
    g_shape_init = true;
}
}  // namespace

StreamShape chidg::stream_shape_for(int kind, int max_b, int esz, bool diagonal) {
    std::lock_guard<std::mutex> lk(g_shape_mu);
    if (!g_shape_init) init_shapes();
    const int c = shape_class(max_b);
    const StreamShape& sh = g_shape[kind][c][width_slot(esz)];
    if (diagonal && sh.standard && kind == kShapeBackward) return StreamShape{8, 2, 24 * 1024, true};
    if (diagonal && sh.standard && kind == kShapeBackwardMv && c == 0) return StreamShape{8, 2, 20 * 1024, true};
    return sh;
}
void chidg::set_stream_shape(int kind, int max_b, int esz, const StreamShape& sh) {
    std::lock_guard<std::mutex> lk(g_shape_mu);
    if (!g_shape_init) init_shapes();
    const int c = shape_class(max_b), w = width_slot(esz);
    StreamShape& at = g_shape[kind][c][w];
    at = sh;
    // the default set again (read, other shapes tried, put back) is the default
    const StreamShape& d = g_default[kind][c][w];
    at.standard = d.standard && sh.cw == d.cw && sh.nstage == d.nstage && sh.stage_bytes == d.stage_bytes;
}
int chidg::resident_ctas(const void* func, int threads, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<int, const void*, int, size_t>, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    auto key = std::make_tuple(dev, func, threads, smem);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, func, threads, smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 0;
    }
    cache[key] = per_sm;
    return per_sm;
}

template <typename TL, typename TU, typename TV, bool FWD, int CW, typename TA = double, bool MV = false>
static int stream_launch(chidg_gpu_precon* M, const TL* LD, const TU* U, StreamTasks Tk, int ntask, const TV* v, TV* zx,
                         void* part, SweepSync S, const StreamShape& sh, int variant, FusedMv<TA, TV> F = {},
                         int mv_cols = 0) {
    chidg_gpu_ctx* ctx = M->ctx;
    using ACC = typename AccOf<TV>::type;
    const int xcols = std::max({M->P.max_b, M->P.max_row_task_cols, mv_cols});    // the widest segment staged in shared memory
    // a stage must hold one column of the widest block (plus the 16-byte rounding)
    if ((size_t)sh.stage_bytes < (size_t)M->P.max_b * std::max(sizeof(TL), sizeof(TU)) + 16 ||
        (MV && (size_t)sh.stage_bytes < (size_t)M->P.max_b * sizeof(TA) + 16))
        return fail(ctx, CHIDG_GPU_EINVAL, "streamed sweep: stage smaller than one block column");
    // a default ring gives way to a very wide staged segment (a row of some 200 blocks)
    constexpr size_t kMostSmem = 226 * 1024;         // beside the kernel's own few hundred bytes
    StreamShape ring = sh;
    auto bytes = [&]() { return stream_smem_bytes(sizeof(ACC), ring.nstage, ring.stage_bytes, xcols, 32 * CW); };
    while (ring.standard && bytes() > kMostSmem && ring.nstage > 2) --ring.nstage;
    if (ring.standard && bytes() > kMostSmem) ring.stage_bytes = std::min(ring.stage_bytes, 20 * 1024);
    const size_t smem = bytes();
    auto k = k_ilu_stream<TL, TU, TV, ACC, FWD, CW, TA, MV>;
    int st;
    if ((st = raise_smem_limit((const void*)k, smem))) return fail(ctx, st, "streamed sweep shared memory");
    const int per_sm = resident_ctas((const void*)k, 32 * CW + 32, smem);
    if (per_sm < 1) return fail(ctx, CHIDG_GPU_EINVAL, "streamed sweep: shape does not fit an SM");
    const int grid = per_sm * ctx->nsm;
    (void)variant;
    // ILU0 and Jacobi: programme row r is matrix row r
    const bool rows_match = (M->kind == CHIDG_PRECON_ILU0 || M->kind == CHIDG_PRECON_JACOBI) && M->P.nprow == ctx->row_mask.nrow;
    const RowMask mk = rows_match ? ctx->row_mask : RowMask{};
    k<<<std::max(1, std::min(grid, ntask)), 32 * CW + 32, smem, ctx->stream>>>(M->P.rows, LD, U, Tk, ntask, v, zx, (ACC*)part,
                                                                              S, ring.nstage, ring.stage_bytes, xcols, F, mk);
    return check_launch(ctx, MV ? "k_ilu_stream backward + matvec" : FWD ? "k_ilu_stream forward" : "k_ilu_stream backward");
}

// Task list of the backward sweep with the matvec rows of A in it: the
// streamed backward sweep's tasks in their order (the keys of stream_tasks,
// scaled by 4), and for every matrix row r a task (r, SW_MATVEC) keyed after the
// last tasks of the last row its columns read, `lag` levels later, so that
// when a CTA takes it the rows it waits for are most likely published.  A
// matvec task waits only for tasks with smaller tickets (deadlock freedom as
// for the sweep).  Needs programme rows == matrix rows (ILU0, Jacobi).
static int build_bwd_mv_tasks(chidg_gpu_precon* M, const chidg_gpu_matrix* A, int lag) {
    IluProgram& P = M->P;
    if (P.bmv_uid == A->uid && P.bmv_lag == lag) return CHIDG_GPU_OK;
    std::vector<int> mv_key;
    mv_key.reserve((size_t)A->nrow);
    std::vector<int32_t> col_prow;
    col_prow.reserve(A->nblk);
    // the matrix blocks that are the sweep's U blocks (same values, same
    // column segment), whose partials a matvec row reuses; reuse only when
    // every U entry of every row is one of its row's blocks
    std::vector<uint8_t> skip;
    skip.reserve(A->nblk);
    bool reuse = true;
    for (int r = 0; r < A->nrow; ++r) {
        int last = -1, matched = 0;
        for (int32_t k : A->rowblk[r]) {
            const int c = A->row(A->ce[k], A->ct[k]);
            col_prow.push_back(c);
            last = std::max(last, 2 * P.lb[c] - 1);
            uint8_t u = 0;
            for (const IluEntry& en : P.up[r])
                if (en.a_off == A->voff[k] && en.parent == c && en.nc == A->bsize(A->ce[k]) &&
                    P.z_off[c] == A->seg(A->ce[k], A->ct[k]))
                    u = 1;
            matched += u;
            skip.push_back(u);
        }
        if (matched != (int)P.up[r].size()) reuse = false;
        mv_key.push_back(4 * (last + 2 * lag) + 2);
    }
    KeyedTasks keyed(-4);
    stream_tasks(P, false, P.lb, 4, 2 * M->ctx->nsm, keyed, &mv_key);
    int st;
    if ((st = upload_items(M->ctx, P.d_bmv_task, keyed.task.get(), (size_t)keyed.n)) || (st = upload_array(M->ctx, P.d_col_prow, col_prow)) ||
        (st = upload_array(M->ctx, P.d_mv_skip, skip)))
        return st;
    P.bmv_reuse = reuse;
    P.ntask_bmv = (int)keyed.n;
    P.bmv_uid = A->uid;
    P.bmv_lag = lag;
    return CHIDG_GPU_OK;
}

// Levels by which a matvec row trails the last row it reads in the fused
// backward sweep; CHIDG_FUSED_MV=0 turns the fusion off (comparison runs),
// CHIDG_FUSED_LAG=<n> sets the lag.
static bool fused_mv_enabled() {
    static const bool v = [] {
        const char* e = std::getenv("CHIDG_FUSED_MV");
        return !(e && e[0] == '0');
    }();
    return v;
}
// CHIDG_FUSED_REUSE=0: the fused matvec rows stream every block instead of
// reusing the sweep's U partials (comparison runs)
static bool fused_reuse_enabled() {
    static const bool v = [] {
        const char* e = std::getenv("CHIDG_FUSED_REUSE");
        return !(e && e[0] == '0');
    }();
    return v;
}
static int fused_mv_lag() {
    static const int v = [] {
        int lag = 1;
        if (const char* e = std::getenv("CHIDG_FUSED_LAG")) lag = std::max(0, std::min(8, std::atoi(e)));
        return lag;
    }();
    return v;
}

// Both sweeps as two streamed launches (CHIDG_SCHED_STREAM): persistent CTAs,
// blocks prefetched into shared memory by a producer lane.  With F, the
// backward launch also runs the matvec rows of F (task list d_bmv_*).
template <typename TL, typename TU, typename TV, typename TA = double>
static int stream_sweeps(chidg_gpu_precon* M, const TL* LD, const TU* U, const TV* v, TV* zx, int variant,
                         const FusedMv<TA, TV>* F = nullptr, int mv_cols = 0, int which = 3) {
    chidg_gpu_ctx* ctx = M->ctx;
    IluProgram& P = M->P;
    using ACC = typename AccOf<TV>::type;
    constexpr int esz = (int)sizeof(TL);
    const StreamShape sh = stream_shape_for(kShapeForward, P.max_b, esz);
    const StreamShape shb = stream_shape_for(F ? kShapeBackwardMv : kShapeBackward, P.max_b, esz, P.diagonal);
    Buffer& pb = (sizeof(ACC) == 8) ? M->part64 : M->part32;
    int st = ensure(ctx, pb, sizeof(ACC) * (size_t)P.part_s);
    if (st) return st;
    // tickets, flags and counts start at zero in every call (also when it is
    // replayed from a graph); a flag is set to a value no host epoch reaches
    constexpr unsigned kStreamEpoch = 0xF0000001u;
    unsigned* sync = (unsigned*)M->sync.ptr;
    unsigned* rowsync = sync + 2;
    const size_t np = (size_t)P.nprow;
    SweepSync S{sync, rowsync, kStreamEpoch, (int*)(ctx->d_scal + kSlotStatus), kSpinLimit};
    cudaError_t e = cudaMemsetAsync(sync, 0, sizeof(unsigned) * (2 + 5 * np), ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "sweep counters");
    int ph = prof_begin(ctx, sizeof(TV) == 8 ? kProfIluForward : kProfIlu32);
    // without lower entries (Jacobi, HB) the backward sweep reads v itself
    if ((which & 1) && !P.no_lower) {
        const StreamTasks Tf{(const StreamTask*)P.d_sf_task.ptr, rowsync + np, nullptr};
        switch (sh.cw) {
            case 16: st = stream_launch<TL, TU, TV, true, 16>(M, LD, U, Tf, P.ntask_sf, v, zx, pb.ptr, S, sh, variant); break;
            case 4: st = stream_launch<TL, TU, TV, true, 4>(M, LD, U, Tf, P.ntask_sf, v, zx, pb.ptr, S, sh, variant); break;
            default: st = stream_launch<TL, TU, TV, true, 8>(M, LD, U, Tf, P.ntask_sf, v, zx, pb.ptr, S, sh, variant);
        }
        if (st) return st;
    }
    if (!(which & 2)) {
        prof_end(ctx, ph);
        return CHIDG_GPU_OK;
    }
    if (sizeof(TV) == 8) {
        prof_end(ctx, ph);
        ph = prof_begin(ctx, F ? kProfIluBackwardMv : kProfIluBackward);
    }
    S.flags = rowsync + 2 * np;
    S.counter = sync + 1;
    if (F) {
        const StreamTasks Tm{(const StreamTask*)P.d_bmv_task.ptr, rowsync + 3 * np, rowsync + 4 * np};
        // the sweep's U partials stand for the matvec's U blocks only when
        // the sweep reads the matvec's own values
        FusedMv<TA, TV> Fr = *F;
        Fr.skip = (P.bmv_reuse && fused_reuse_enabled() && sizeof(TU) == sizeof(TA) &&
                   (const void*)U == (const void*)F->val)
                      ? (const uint8_t*)P.d_mv_skip.ptr
                      : nullptr;
        switch (shb.cw) {
            case 16: st = stream_launch<TL, TU, TV, false, 16, TA, true>(M, LD, U, Tm, P.ntask_bmv, v, zx, pb.ptr, S, shb, variant, Fr, mv_cols); break;
            case 4: st = stream_launch<TL, TU, TV, false, 4, TA, true>(M, LD, U, Tm, P.ntask_bmv, v, zx, pb.ptr, S, shb, variant, Fr, mv_cols); break;
            default: st = stream_launch<TL, TU, TV, false, 8, TA, true>(M, LD, U, Tm, P.ntask_bmv, v, zx, pb.ptr, S, shb, variant, Fr, mv_cols);
        }
        if (st) return st;
        prof_end(ctx, ph);
        return CHIDG_GPU_OK;
    }
    const StreamTasks Tb{(const StreamTask*)P.d_sb_task.ptr, rowsync + 3 * np, rowsync + 4 * np};
    switch (shb.cw) {
        case 16: st = stream_launch<TL, TU, TV, false, 16>(M, LD, U, Tb, P.ntask_sb, v, zx, pb.ptr, S, shb, variant); break;
        case 4: st = stream_launch<TL, TU, TV, false, 4>(M, LD, U, Tb, P.ntask_sb, v, zx, pb.ptr, S, shb, variant); break;
        default: st = stream_launch<TL, TU, TV, false, 8>(M, LD, U, Tb, P.ntask_sb, v, zx, pb.ptr, S, shb, variant);
    }
    if (st) return st;
    prof_end(ctx, ph);
    return CHIDG_GPU_OK;
}

extern "C" int chidg_gpu_precon_set_schedule(chidg_gpu_precon* M, int32_t schedule) {
    if (!M || schedule < CHIDG_SCHED_LEVELS || schedule > CHIDG_SCHED_STREAM) return CHIDG_GPU_EINVAL;
    M->schedule = schedule;
    return CHIDG_GPU_OK;
}

template <typename TV>
int chidg::precon_apply_impl(chidg_gpu_precon* M, const TV* v, TV* z, int precision) {
    chidg_gpu_ctx* ctx = M->ctx;
    chidg_gpu_matrix* A = M->A;
    const int64_t n = A->n;
    if (M->kind == CHIDG_PRECON_IDENTITY) {
        const cudaError_t e = cudaMemcpyAsync(z, v, sizeof(TV) * (size_t)n, cudaMemcpyDeviceToDevice, ctx->stream);
        return e == cudaSuccess ? CHIDG_GPU_OK : cuda_fail(ctx, e, "identity apply");
    }
    int st0;
    if ((st0 = precon_source(M, &A))) return st0;     // the U blocks come from A^T for a transposed A
    IluProgram& P = M->P;
    using ACC = typename AccOf<TV>::type;
    // work buffer: the output itself when there are no overlap rows
    TV* zx = z;
    if (P.n_ext != n) {
        Buffer& wb = (sizeof(TV) == 8) ? M->zx : M->zx32;
        int st = ensure(ctx, wb, sizeof(TV) * (size_t)P.n_ext);
        if (st) return st;
        zx = (TV*)wb.ptr;
    }
    const int threads = P.sweep_threads;
    const size_t smem_f = sizeof(ACC) * ((size_t)P.max_lo_cols + threads) + 512;
    const size_t smem_b = sizeof(ACC) * ((size_t)P.max_up_cols + P.max_b + threads) + 512;
    const int nf = (int)P.fwd_ptr.size() - 1, nb = (int)P.bwd_ptr.size() - 1;
    int st;
    // blocks of more than 1024 rows: the streamed sweeps run as TASKS
    const int sched = (M->schedule == CHIDG_SCHED_STREAM && P.max_b > SS_MAX_B) ? CHIDG_SCHED_TASKS : M->schedule;
    if (sizeof(TV) == 8 && precision == CHIDG_GPU_MIXED_PRECON_FP32) {
        // FP64 vectors and accumulation, FP32 blocks (streamed or task sweeps)
        int st = (sched == CHIDG_SCHED_STREAM)
                     ? stream_sweeps(M, (const float*)M->LD32.ptr, (const float*)A->val32.ptr, v, zx, 3)
                     : task_sweeps(M, (const float*)M->LD32.ptr, (const float*)A->val32.ptr, v, zx, 3);
        if (st) return st;
        if (zx != z) {
            const cudaError_t e = cudaMemcpyAsync(z, zx, sizeof(TV) * (size_t)n, cudaMemcpyDeviceToDevice, ctx->stream);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "precon output copy");
        }
        return CHIDG_GPU_OK;
    }
    if (sched == CHIDG_SCHED_STREAM) {
        int st;
        if (precision == CHIDG_GPU_MIXED_BF16 && sizeof(TV) == 4)
            st = stream_sweeps(M, (const __nv_bfloat16*)M->LD16.ptr, (const __nv_bfloat16*)A->val16.ptr, v, zx, 2);
        else if (sizeof(TV) == 4)
            st = stream_sweeps(M, (const float*)M->LD32.ptr, (const float*)A->val32.ptr, v, zx, 1);
        else
            st = stream_sweeps(M, (const double*)M->LD.ptr, (const double*)A->val.ptr, v, zx, 0);
        if (st) return st;
        if (zx != z) {
            const cudaError_t e = cudaMemcpyAsync(z, zx, sizeof(TV) * (size_t)n, cudaMemcpyDeviceToDevice, ctx->stream);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "precon output copy");
        }
        return CHIDG_GPU_OK;
    }
    if (sched == CHIDG_SCHED_DATAFLOW || sched == CHIDG_SCHED_TASKS) {
        const bool tk = sched == CHIDG_SCHED_TASKS;
        if (precision == CHIDG_GPU_MIXED_BF16 && sizeof(TV) == 4)
            st = tk ? task_sweeps(M, (const __nv_bfloat16*)M->LD16.ptr, (const __nv_bfloat16*)A->val16.ptr, v, zx, 2)
                    : dataflow_sweeps(M, (const __nv_bfloat16*)M->LD16.ptr, (const __nv_bfloat16*)A->val16.ptr, v, zx, 2);
        else if (sizeof(TV) == 4)
            st = tk ? task_sweeps(M, (const float*)M->LD32.ptr, (const float*)A->val32.ptr, v, zx, 1)
                    : dataflow_sweeps(M, (const float*)M->LD32.ptr, (const float*)A->val32.ptr, v, zx, 1);
        else
            st = tk ? task_sweeps(M, (const double*)M->LD.ptr, (const double*)A->val.ptr, v, zx, 0)
                    : dataflow_sweeps(M, (const double*)M->LD.ptr, (const double*)A->val.ptr, v, zx, 0);
        if (st) return st;
        if (zx != z) {
            const cudaError_t e = cudaMemcpyAsync(z, zx, sizeof(TV) * (size_t)n, cudaMemcpyDeviceToDevice, ctx->stream);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "precon output copy");
        }
        return CHIDG_GPU_OK;
    }
    int ph = prof_begin(ctx, sizeof(TV) == 8 ? kProfIluForward : kProfIlu32);
    for (int l = 0; l < nf; ++l) {
        const int cnt = P.fwd_ptr[l + 1] - P.fwd_ptr[l];
        if (precision == CHIDG_GPU_MIXED_BF16 && sizeof(TV) == 4)
            k_ilu_forward<__nv_bfloat16, TV, ACC><<<cnt, threads, smem_f, ctx->stream>>>(P.rows, (const __nv_bfloat16*)M->LD16.ptr, (const int32_t*)P.d_fwd_rows.ptr, P.fwd_ptr[l], v, zx);
        else if (sizeof(TV) == 4)
            k_ilu_forward<float, TV, ACC><<<cnt, threads, smem_f, ctx->stream>>>(P.rows, (const float*)M->LD32.ptr, (const int32_t*)P.d_fwd_rows.ptr, P.fwd_ptr[l], v, zx);
        else
            k_ilu_forward<double, TV, ACC><<<cnt, threads, smem_f, ctx->stream>>>(P.rows, (const double*)M->LD.ptr, (const int32_t*)P.d_fwd_rows.ptr, P.fwd_ptr[l], v, zx);
        if ((st = check_launch(ctx, "k_ilu_forward"))) return st;
    }
    if (sizeof(TV) == 8) {
        prof_end(ctx, ph);
        ph = prof_begin(ctx, kProfIluBackward);
    }
    for (int l = 0; l < nb; ++l) {
        const int cnt = P.bwd_ptr[l + 1] - P.bwd_ptr[l];
        if (precision == CHIDG_GPU_MIXED_BF16 && sizeof(TV) == 4)
            k_ilu_backward<__nv_bfloat16, __nv_bfloat16, TV, ACC><<<cnt, threads, smem_b, ctx->stream>>>(P.rows, (const __nv_bfloat16*)M->LD16.ptr, (const __nv_bfloat16*)A->val16.ptr, (const int32_t*)P.d_bwd_rows.ptr, P.bwd_ptr[l], zx);
        else if (sizeof(TV) == 4)
            k_ilu_backward<float, float, TV, ACC><<<cnt, threads, smem_b, ctx->stream>>>(P.rows, (const float*)M->LD32.ptr, (const float*)A->val32.ptr, (const int32_t*)P.d_bwd_rows.ptr, P.bwd_ptr[l], zx);
        else
            k_ilu_backward<double, double, TV, ACC><<<cnt, threads, smem_b, ctx->stream>>>(P.rows, (const double*)M->LD.ptr, (const double*)A->val.ptr, (const int32_t*)P.d_bwd_rows.ptr, P.bwd_ptr[l], zx);
        if ((st = check_launch(ctx, "k_ilu_backward"))) return st;
    }
    prof_end(ctx, ph);
    if (zx != z) {
        const cudaError_t e = cudaMemcpyAsync(z, zx, sizeof(TV) * (size_t)n, cudaMemcpyDeviceToDevice, ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "precon output copy");
    }
    return CHIDG_GPU_OK;
}
template int chidg::precon_apply_impl<double>(chidg_gpu_precon*, const double*, double*, int);
template int chidg::precon_apply_impl<float>(chidg_gpu_precon*, const float*, float*, int);

template <typename TV, typename TA>
int chidg::precon_apply_mv(chidg_gpu_precon* M, const TV* v, TV* z, int precision, chidg_gpu_matrix* Aop, const TA* val,
                           TV* w, double* row_sq) {
    constexpr int kNotFused = 1;
    if (!fused_mv_enabled() || !(M->kind == CHIDG_PRECON_ILU0 || M->kind == CHIDG_PRECON_JACOBI)) return kNotFused;
    // the matvec's value type must be the one the solver's product reads
    constexpr bool ta_bf16 = std::is_same<TA, __nv_bfloat16>::value;
    if (sizeof(TV) == 4 && ta_bf16 != (precision == CHIDG_GPU_MIXED_BF16)) return kNotFused;
    chidg_gpu_matrix* S = nullptr;
    int st;
    if ((st = precon_source(M, &S))) return st;
    IluProgram& P = M->P;
    if (S != Aop || M->schedule != CHIDG_SCHED_STREAM || P.max_b > SS_MAX_B || P.n_ext != Aop->n ||
        P.nprow != Aop->nrow || !Aop->rows_contiguous || Aop->max_b > SS_MAX_B || matvec_rows_env())
        return kNotFused;
    if ((st = build_bwd_mv_tasks(M, Aop, fused_mv_lag()))) return st;
    MatvecRowsView R{(const int64_t*)Aop->d_row_ptr.ptr, (const int64_t*)Aop->d_blk_voff.ptr,
                     (const int64_t*)Aop->d_blk_xoff.ptr, (const int32_t*)Aop->d_blk_nc.ptr,
                     (const int64_t*)Aop->d_row_yoff.ptr, (const int32_t*)Aop->d_row_b.ptr};
    const FusedMv<TA, TV> F{R, val, w, row_sq, (const int32_t*)P.d_col_prow.ptr};
    if constexpr (sizeof(TV) == 8) {
        if (precision == CHIDG_GPU_MIXED_PRECON_FP32)
            return stream_sweeps(M, (const float*)M->LD32.ptr, (const float*)S->val32.ptr, v, z, 3, &F, Aop->max_row_cols);
        return stream_sweeps(M, (const double*)M->LD.ptr, (const double*)S->val.ptr, v, z, 0, &F, Aop->max_row_cols);
    } else {
        if (precision == CHIDG_GPU_MIXED_BF16)
            return stream_sweeps(M, (const __nv_bfloat16*)M->LD16.ptr, (const __nv_bfloat16*)S->val16.ptr, v, z, 2, &F,
                                 Aop->max_row_cols);
        return stream_sweeps(M, (const float*)M->LD32.ptr, (const float*)S->val32.ptr, v, z, 1, &F, Aop->max_row_cols);
    }
}
template int chidg::precon_apply_mv<double, double>(chidg_gpu_precon*, const double*, double*, int, chidg_gpu_matrix*,
                                                    const double*, double*, double*);
template int chidg::precon_apply_mv<float, float>(chidg_gpu_precon*, const float*, float*, int, chidg_gpu_matrix*,
                                                  const float*, float*, double*);
template int chidg::precon_apply_mv<float, __nv_bfloat16>(chidg_gpu_precon*, const float*, float*, int, chidg_gpu_matrix*,
                                                          const __nv_bfloat16*, float*, double*);

int chidg::precon_set_smem(chidg_gpu_precon* M) {
    IluProgram& P = M->P;
    const int threads = P.sweep_threads;
    const size_t sf = sizeof(double) * ((size_t)P.max_lo_cols + threads) + 512;
    const size_t sb = sizeof(double) * ((size_t)P.max_up_cols + P.max_b + threads) + 512;
    int st;
    if ((st = raise_smem_limit((const void*)k_ilu_forward<double, double, double>, sf)) ||
        (st = raise_smem_limit((const void*)k_ilu_forward<float, float, float>, sf)) ||
        (st = raise_smem_limit((const void*)k_ilu_forward<__nv_bfloat16, float, float>, sf)) ||
        (st = raise_smem_limit((const void*)k_ilu_backward<double, double, double, double>, sb)) ||
        (st = raise_smem_limit((const void*)k_ilu_backward<float, float, float, float>, sb)) ||
        (st = raise_smem_limit((const void*)k_ilu_backward<__nv_bfloat16, __nv_bfloat16, float, float>, sb)))
        return st;
    return CHIDG_GPU_OK;
}

extern "C" int chidg_gpu_precon_apply(chidg_gpu_precon* M, chidg_gpu_matrix* A, const chidg_gpu_vector* v, chidg_gpu_vector* z) {
    if (!M || !A || !v || !z || A != M->A || v->n != A->n || z->n != A->n || v == z) return CHIDG_GPU_EINVAL;
    cudaSetDevice(M->ctx->device);
    if (M->kind != CHIDG_PRECON_IDENTITY && M->stamp == 0) return fail(M->ctx, CHIDG_GPU_ESTATE, "precon_apply: preconditioner not updated");
    if (M->kind != CHIDG_PRECON_IDENTITY && !M->ld64_valid)
        return fail(M->ctx, CHIDG_GPU_ESTATE, "precon_apply: the factors were computed in FP32 (mixed precision); update in FP64 first");
    precon_set_smem(M);
    chidg_gpu_ctx* ctx = M->ctx;
    cudaMemsetAsync(ctx->d_scal + kSlotStatus, 0, sizeof(double), ctx->stream);
    int st = precon_apply_impl<double>(M, (const double*)v->buf.ptr, (double*)z->buf.ptr, CHIDG_GPU_FP64);
    if (st) return st;
    double w;
    if ((st = fetch_scalars(ctx, kSlotStatus, 1, &w))) return st;
    return status_word(ctx, w);
}

// The factors in the matrix's block positions, from LD (FP64) or LD32 (FP32)
template <typename T>
static int download_factors(chidg_gpu_precon* M, T* host, const Buffer& src, bool valid, const char* what) {
    if (!M || !host) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = M->ctx;
    cudaSetDevice(ctx->device);
    chidg_gpu_matrix* A = M->A;
    if (M->kind == CHIDG_PRECON_IDENTITY || M->stamp == 0) return fail(ctx, CHIDG_GPU_ESTATE, std::string(what) + ": no factors");
    if (!valid || !src.ptr) return fail(ctx, CHIDG_GPU_ESTATE, std::string(what) + ": no factors of this precision since the last update");
    if (M->kind == CHIDG_PRECON_HB)
        return fail(ctx, CHIDG_GPU_EINVAL, std::string(what) + ": the HB preconditioner's element blocks span time levels");
    if (M->kind != CHIDG_PRECON_RASILU0 && M->built_transposed) A = A->T;   // factors of A^T, in A^T's block order
    std::vector<T> ld((size_t)M->P.ld_size);
    cudaError_t e = cudaMemcpyAsync(ld.data(), src.ptr, sizeof(T) * ld.size(), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "LD download");
    std::memset(host, 0, sizeof(T) * (size_t)A->nval);
    const IluProgram& P = M->P;
    for (int pr = 0; pr < P.nprow; ++pr) {
        if (P.diag_blk[pr] < 0) continue;   // overlap rows live only inside the preconditioner
        const int b = P.prow_b[pr];
        std::memcpy(host + A->voff[P.diag_blk[pr]], ld.data() + P.dinv_off[pr], sizeof(T) * b * b);
        for (const auto& en : P.lo[pr])
            if (en.blk >= 0) std::memcpy(host + A->voff[en.blk], ld.data() + en.l_off, sizeof(T) * (size_t)b * en.nc);
    }
    return CHIDG_GPU_OK;
}

extern "C" int chidg_gpu_precon_download_LD(chidg_gpu_precon* M, double* host) {
    if (M && M->stamp != 0 && !M->ld64_valid)
        return fail(M->ctx, CHIDG_GPU_ESTATE, "download_LD: the factors were computed in FP32 (mixed precision)");
    return M ? download_factors<double>(M, host, M->LD, M->ld64_valid, "download_LD") : CHIDG_GPU_EINVAL;
}

extern "C" int chidg_gpu_precon_download_LD32(chidg_gpu_precon* M, float* host) {
    if (!M) return CHIDG_GPU_EINVAL;
    // BF16 factors come through FP32 ones only on the FP32 factorisation's path
    const bool fp32 = M->precision == CHIDG_GPU_MIXED_FP32 || M->precision == CHIDG_GPU_MIXED_PRECON_FP32 ||
                      (M->precision == CHIDG_GPU_MIXED_BF16 && M->P.max_b <= SF_MAX && !M->P.assembled);
    return download_factors<float>(M, host, M->LD32, fp32, "download_LD32");
}

// ---------------------------------------------------------------------------
// Autotuner of the streamed kernels' launch shapes
// ---------------------------------------------------------------------------
namespace {
__global__ void k_fill(double* x, int64_t n, double v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) x[i] = v;
}
__global__ void k_fill32(float* x, int64_t n, float v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) x[i] = v;
}
}  // namespace

// Candidate shapes: 4, 8 or 16 consumer warps; 2 to 4 stages of 8 to 48 KB
// (ring at most 104 KB); a stage holds at least one column of the widest block.
static std::vector<StreamShape> shape_candidates(int max_b, int esz) {
    std::vector<StreamShape> out;
    for (int cw : {4, 8, 16})
        for (int ns : {2, 3, 4})
            for (int kb : {8, 12, 16, 20, 24, 25, 26, 32, 40, 48}) {
                if (ns * kb > 104) continue;
                if ((size_t)kb * 1024 < (size_t)max_b * esz + 16) continue;
                out.push_back(StreamShape{cw, ns, kb * 1024});
            }
    return out;
}

extern "C" int chidg_gpu_autotune(chidg_gpu_precon* M, chidg_gpu_matrix* A, int32_t precision, int32_t reps) {
    if (!M || !A || M->A != A || reps < 1 || reps > 100) return CHIDG_GPU_EINVAL;
    chidg_gpu_ctx* ctx = M->ctx;
    cudaSetDevice(ctx->device);
    if (precision != CHIDG_GPU_FP64 && precision != CHIDG_GPU_MIXED_PRECON_FP32 && precision != CHIDG_GPU_MIXED_FP32 &&
        precision != CHIDG_GPU_MIXED_BF16)
        return fail(ctx, CHIDG_GPU_EINVAL, "autotune: bad precision");
    if (M->kind == CHIDG_PRECON_IDENTITY || M->stamp == 0 || M->precision != precision)
        return fail(ctx, CHIDG_GPU_ESTATE, "autotune: update the preconditioner for A in this precision first");
    if (M->schedule != CHIDG_SCHED_STREAM || M->P.max_b > SS_MAX_B)
        return fail(ctx, CHIDG_GPU_EINVAL, "autotune: the streamed schedule only");
    chidg_gpu_matrix* Aop = nullptr;
    int st;
    if ((st = matrix_op(A, &Aop))) return st;
    if ((st = matrix_lowp(Aop, precision))) return st;
    precon_set_smem(M);
    const bool lowp_vec = precision == CHIDG_GPU_MIXED_FP32 || precision == CHIDG_GPU_MIXED_BF16;
    const int esz_blocks = precision == CHIDG_GPU_FP64 ? 8 : precision == CHIDG_GPU_MIXED_BF16 ? 2 : 4;
    const int esz_matvec = precision == CHIDG_GPU_MIXED_PRECON_FP32 ? 8 : esz_blocks;
    const int64_t n = std::max<int64_t>(M->P.n_ext, Aop->n);
    Buffer bv, bz, bw, brs;
    auto cleanup = [&]() { for (Buffer* b : {&bv, &bz, &bw, &brs}) release(*b); };
    const size_t vb = (lowp_vec ? sizeof(float) : sizeof(double)) * (size_t)n;
    if ((st = ensure(ctx, bv, vb)) || (st = ensure(ctx, bz, vb)) || (st = ensure(ctx, bw, vb)) ||
        (st = ensure(ctx, brs, sizeof(double) * (size_t)Aop->nrow))) {
        cleanup();
        return st;
    }
    if (lowp_vec) k_fill32<<<ctx->nsm * 4, 256, 0, ctx->stream>>>((float*)bv.ptr, n, 1.0f);
    else k_fill<<<ctx->nsm * 4, 256, 0, ctx->stream>>>((double*)bv.ptr, n, 1.0);
    cudaMemsetAsync(bz.ptr, 0, vb, ctx->stream);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const bool prof = ctx->profiling;
    ctx->profiling = false;
    cudaMemsetAsync(ctx->d_scal + kSlotStatus, 0, sizeof(double), ctx->stream);
    // one run of the kernel kind, launched with the table's current shape
    auto run_kind = [&](int kind) -> int {
        if (!lowp_vec) {
            const double* v = (const double*)bv.ptr;
            double* z = (double*)bz.ptr;
            double* w = (double*)bw.ptr;
            if (kind == kShapeMatvec) return matvec_launch<double, double>(Aop, (const double*)Aop->val.ptr, z, w, nullptr, 1.0, 0.0, (double*)brs.ptr);
            const bool p32 = precision == CHIDG_GPU_MIXED_PRECON_FP32;
            chidg_gpu_matrix* S = nullptr;
            int s2 = precon_source(M, &S);
            if (s2) return s2;
            if (kind == kShapeBackwardMv) {
                if (M->kind != CHIDG_PRECON_ILU0 && M->kind != CHIDG_PRECON_JACOBI) return 1;
                if (S != Aop || M->P.n_ext != Aop->n || M->P.nprow != Aop->nrow || !Aop->rows_contiguous) return 1;
                if ((s2 = build_bwd_mv_tasks(M, Aop, fused_mv_lag()))) return s2;
                MatvecRowsView R{(const int64_t*)Aop->d_row_ptr.ptr, (const int64_t*)Aop->d_blk_voff.ptr,
                                 (const int64_t*)Aop->d_blk_xoff.ptr, (const int32_t*)Aop->d_blk_nc.ptr,
                                 (const int64_t*)Aop->d_row_yoff.ptr, (const int32_t*)Aop->d_row_b.ptr};
                const FusedMv<double, double> F{R, (const double*)Aop->val.ptr, w, (double*)brs.ptr, (const int32_t*)M->P.d_col_prow.ptr};
                return p32 ? stream_sweeps(M, (const float*)M->LD32.ptr, (const float*)S->val32.ptr, v, z, 3, &F, Aop->max_row_cols, 2)
                           : stream_sweeps(M, (const double*)M->LD.ptr, (const double*)S->val.ptr, v, z, 0, &F, Aop->max_row_cols, 2);
            }
            const int which = kind == kShapeForward ? 1 : 2;
            return p32 ? stream_sweeps<float, float, double>(M, (const float*)M->LD32.ptr, (const float*)S->val32.ptr, v, z, 3, (const FusedMv<double, double>*)nullptr, 0, which)
                       : stream_sweeps<double, double, double>(M, (const double*)M->LD.ptr, (const double*)S->val.ptr, v, z, 0, (const FusedMv<double, double>*)nullptr, 0, which);
        }
        const float* v = (const float*)bv.ptr;
        float* z = (float*)bz.ptr;
        float* w = (float*)bw.ptr;
        chidg_gpu_matrix* S = nullptr;
        int s2 = precon_source(M, &S);
        if (s2) return s2;
        const bool bf = precision == CHIDG_GPU_MIXED_BF16;
        if (kind == kShapeMatvec)
            return bf ? matvec_launch<__nv_bfloat16, float>(Aop, (const __nv_bfloat16*)Aop->val16.ptr, z, w, nullptr, 1.0, 0.0, (double*)brs.ptr)
                      : matvec_launch<float, float>(Aop, (const float*)Aop->val32.ptr, z, w, nullptr, 1.0, 0.0, (double*)brs.ptr);
        if (kind == kShapeBackwardMv) {
            if (M->kind != CHIDG_PRECON_ILU0 && M->kind != CHIDG_PRECON_JACOBI) return 1;
            if (S != Aop || M->P.n_ext != Aop->n || M->P.nprow != Aop->nrow || !Aop->rows_contiguous) return 1;
            if ((s2 = build_bwd_mv_tasks(M, Aop, fused_mv_lag()))) return s2;
            MatvecRowsView R{(const int64_t*)Aop->d_row_ptr.ptr, (const int64_t*)Aop->d_blk_voff.ptr,
                             (const int64_t*)Aop->d_blk_xoff.ptr, (const int32_t*)Aop->d_blk_nc.ptr,
                             (const int64_t*)Aop->d_row_yoff.ptr, (const int32_t*)Aop->d_row_b.ptr};
            if (bf) {
                const FusedMv<__nv_bfloat16, float> F{R, (const __nv_bfloat16*)Aop->val16.ptr, w, (double*)brs.ptr, (const int32_t*)M->P.d_col_prow.ptr};
                return stream_sweeps(M, (const __nv_bfloat16*)M->LD16.ptr, (const __nv_bfloat16*)S->val16.ptr, v, z, 2, &F, Aop->max_row_cols, 2);
            }
            const FusedMv<float, float> F{R, (const float*)Aop->val32.ptr, w, (double*)brs.ptr, (const int32_t*)M->P.d_col_prow.ptr};
            return stream_sweeps(M, (const float*)M->LD32.ptr, (const float*)S->val32.ptr, v, z, 1, &F, Aop->max_row_cols, 2);
        }
        const int which = kind == kShapeForward ? 1 : 2;
        return bf ? stream_sweeps<__nv_bfloat16, __nv_bfloat16, float>(M, (const __nv_bfloat16*)M->LD16.ptr, (const __nv_bfloat16*)S->val16.ptr, v, z, 2, (const FusedMv<double, float>*)nullptr, 0, which)
                  : stream_sweeps<float, float, float>(M, (const float*)M->LD32.ptr, (const float*)S->val32.ptr, v, z, 1, (const FusedMv<double, float>*)nullptr, 0, which);
    };
    for (int kind = 0; kind < kShapeKinds && st == CHIDG_GPU_OK; ++kind) {
        const int max_b = kind == kShapeMatvec ? Aop->max_b : M->P.max_b;
        const int esz = kind == kShapeMatvec ? esz_matvec : esz_blocks;
        if (kind == kShapeMatvec && (Aop->max_b > SS_MAX_B || !Aop->rows_contiguous)) continue;
        if (kind == kShapeForward && M->P.no_lower) continue;     // nothing runs: the class keeps its shape
        const StreamShape keep = stream_shape_for(kind, max_b, esz);
        StreamShape best = keep;
        float best_ms = 1e30f;
        bool any = false;
        for (const StreamShape& cand : shape_candidates(std::max(max_b, kind == kShapeBackwardMv ? Aop->max_b : 0), esz)) {
            set_stream_shape(kind, max_b, esz, cand);
            int s2 = run_kind(kind);                              // warm-up (and the shared-memory limit)
            if (s2 == 1) break;                                   // this kind does not apply here
            if (s2 == CHIDG_GPU_EINVAL) { ctx->err.clear(); continue; }   // does not fit an SM
            if (s2) { st = s2; break; }
            cudaEventRecord(e0, ctx->stream);
            for (int r = 0; r < reps && !s2; ++r) s2 = run_kind(kind);
            cudaEventRecord(e1, ctx->stream);
            if (s2) { st = s2; break; }
            const cudaError_t e = cudaEventSynchronize(e1);
            if (e != cudaSuccess) { st = cuda_fail(ctx, e, "autotune"); break; }
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, e0, e1);
            any = true;
            if (ms < best_ms) { best_ms = ms; best = cand; }
        }
        set_stream_shape(kind, max_b, esz, any ? best : keep);
    }
    ctx->profiling = prof;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st == CHIDG_GPU_OK) {
        double w = 0.0;
        if ((st = fetch_scalars(ctx, kSlotStatus, 1, &w)) == CHIDG_GPU_OK) st = status_word(ctx, w);
    }
    cleanup();
    return st;
}

extern "C" int chidg_gpu_stream_shape_get(int32_t kind, int32_t max_b, int32_t value_bytes, int32_t* warps, int32_t* stages,
                                          int32_t* stage_bytes) {
    if (kind < 0 || kind >= kShapeKinds || max_b < 1 || max_b > SS_MAX_B || !warps || !stages || !stage_bytes ||
        (value_bytes != 8 && value_bytes != 4 && value_bytes != 2))
        return CHIDG_GPU_EINVAL;
    const StreamShape sh = stream_shape_for(kind, max_b, value_bytes);
    *warps = sh.cw;
    *stages = sh.nstage;
    *stage_bytes = sh.stage_bytes;
    return CHIDG_GPU_OK;
}

extern "C" int chidg_gpu_stream_shape_set(int32_t kind, int32_t max_b, int32_t value_bytes, int32_t warps, int32_t stages,
                                          int32_t stage_bytes) {
    if (kind < 0 || kind >= kShapeKinds || max_b < 1 || max_b > SS_MAX_B ||
        (value_bytes != 8 && value_bytes != 4 && value_bytes != 2) || (warps != 4 && warps != 8 && warps != 16) ||
        stages < 2 || stages > SS_MAX_STAGES || stage_bytes < 2048 || stage_bytes > 96 * 1024 || stage_bytes % 16 != 0)
        return CHIDG_GPU_EINVAL;
    set_stream_shape(kind, max_b, value_bytes, StreamShape{warps, stages, stage_bytes});
    return CHIDG_GPU_OK;
}
