// Context, grid and derivative application (K2: ELL SpMV) of librbffd_sm100.
//
// Device layout of a grid: the sliced ELL arrays of ell.cuh (32-row slices,
// 4-slot chunks), n4 = n_pad rounded up to 4 slots per row, rows in the
// grid's internal (Morton) order.  A lane reads four consecutive slots of its
// row with one 16-byte index load and one 16-byte (FP32) or two 16-byte
// (FP64) weight loads.  Padding slots (s >= len[i]) hold the centre index and
// weight 0, as RBFFD_CL's ELL packing does (src/rbffd/rbffd_cl.cpp:238-242,
// 349-353), so every row runs n4 slots without a length check and the extra
// terms add exactly zero.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <cstring>
#include <functional>
#include <iterator>
#include <new>
#include <thread>
#include <type_traits>

#include "ell.cuh"
#include "internal.h"

// ---------------------------------------------------------------------------
// errors and accounting

int set_error(rbffd_ctx* ctx, int status, const char* fmt, ...)
{
    if (ctx) {
        char buf[1024];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof buf, fmt, ap);
        va_end(ap);
        std::lock_guard<std::mutex> lk(ctx->err_mu);
        ctx->last_error = buf;
    }
    return status;
}

KeepError::KeepError(rbffd_ctx* c) : ctx(c)
{
    std::lock_guard<std::mutex> lk(ctx->err_mu);
    msg = ctx->last_error;
}
KeepError::~KeepError()
{
    std::lock_guard<std::mutex> lk(ctx->err_mu);
    if (ctx->last_error != msg) ctx->last_error = msg;
}

int cuda_error(rbffd_ctx* ctx, cudaError_t e, const char* what)
{
    int st = (e == cudaErrorMemoryAllocation) ? RBFFD_ERR_OOM : RBFFD_ERR_CUDA;
    cudaGetLastError();  // clear a sticky non-fatal error so the context stays usable
    return set_error(ctx, st, "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
}

int dev_alloc(rbffd_ctx* ctx, void** p, size_t bytes)
{
    *p = nullptr;
    if (bytes == 0) return RBFFD_OK;
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && ctx_trim(ctx) > 0) {
        cudaGetLastError();
        e = cudaMalloc(p, bytes);
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        return cuda_error(ctx, e, "cudaMalloc");
    }
    std::lock_guard<std::mutex> lk(ctx->mu);
    ctx->held += bytes;
    return RBFFD_OK;
}

void dev_free(rbffd_ctx* ctx, void* p, size_t bytes)
{
    if (!p) return;
    cudaFree(p);
    std::lock_guard<std::mutex> lk(ctx->mu);
    ctx->held -= std::min(ctx->held, bytes);
}

void* keep_take(rbffd_ctx* ctx, Kept* k, size_t bytes)
{
    {
        std::lock_guard<std::mutex> lk(ctx->kept_mu);
        if (!k->listed) ctx->kept.push_back(k);
        k->listed = k->busy = true;
        if (k->bytes >= bytes) return k->p;
        dev_free(ctx, k->p, k->bytes);
        k->p = nullptr;
        k->bytes = 0;
    }
    void* p = nullptr;
    const int rc = dev_alloc(ctx, &p, bytes);
    std::lock_guard<std::mutex> lk(ctx->kept_mu);
    k->p = p;
    k->bytes = rc == RBFFD_OK ? bytes : 0;
    return p;
}

void keep_release(rbffd_ctx* ctx, Kept* k)
{
    std::lock_guard<std::mutex> lk(ctx->kept_mu);
    k->busy = false;
}

void keep_free(rbffd_ctx* ctx, Kept* k)
{
    std::lock_guard<std::mutex> lk(ctx->kept_mu);
    ctx->kept.erase(std::remove(ctx->kept.begin(), ctx->kept.end(), k), ctx->kept.end());
    dev_free(ctx, k->p, k->bytes);
    *k = Kept{};
}

size_t ctx_kept(rbffd_ctx* ctx)
{
    std::lock_guard<std::mutex> lk(ctx->kept_mu);
    size_t sum = 0;
    for (const Kept* k : ctx->kept)
        if (!k->busy) sum += k->bytes;
    return sum;
}

size_t ctx_in_use(rbffd_ctx* ctx)
{
    const size_t kept = ctx_kept(ctx);
    std::lock_guard<std::mutex> lk(ctx->mu);
    return ctx->held - std::min(ctx->held, kept);
}

size_t ctx_trim(rbffd_ctx* ctx)
{
    std::lock_guard<std::mutex> lk(ctx->kept_mu);
    size_t sum = 0;
    for (Kept* k : ctx->kept)
        if (!k->busy && k->p) {
            sum += k->bytes;
            dev_free(ctx, k->p, k->bytes);
            k->p = nullptr;
            k->bytes = 0;
        }
    return sum;
}

extern "C" const char* rbffd_version(void) { return RBFFD_VERSION_STRING; }

extern "C" const char* rbffd_status_string(int s)
{
    switch (s) {
    case RBFFD_OK: return "ok";
    case RBFFD_ERR_INVALID: return "invalid argument";
    case RBFFD_ERR_OOM: return "out of memory";
    case RBFFD_ERR_CUDA: return "CUDA error";
    case RBFFD_ERR_TIMEOUT: return "timeout";
    case RBFFD_ERR_UNSUPPORTED: return "unsupported";
    case RBFFD_ERR_STATE: return "invalid state";
    case RBFFD_ERR_SINGULAR: return "singular stencil system";
    case RBFFD_ERR_BUDGET: return "over device memory budget";
    case RBFFD_ERR_NO_DEVICE: return "no CUDA device";
    case RBFFD_ERR_CANCELLED: return "request cancelled";
    }
    return "unknown status";
}

extern "C" int rbffd_device_count(int* count)
{
    if (!count) return RBFFD_ERR_INVALID;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) {
        cudaGetLastError();
        *count = 0;
        return RBFFD_ERR_NO_DEVICE;
    }
    *count = n;
    return RBFFD_OK;
}

// ---------------------------------------------------------------------------
// context

extern "C" int rbffd_ctx_create(int device, rbffd_ctx** out)
{
    if (!out) return RBFFD_ERR_INVALID;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
        cudaGetLastError();
        return RBFFD_ERR_NO_DEVICE;
    }
    if (device < 0 || device >= n) return RBFFD_ERR_INVALID;
    rbffd_ctx* c = new (std::nothrow) rbffd_ctx();
    if (!c) return RBFFD_ERR_OOM;
    c->device = device;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        delete c;
        return RBFFD_ERR_CUDA;
    }
    cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, device);
    if (cudaMalloc((void**)&c->d_status, sizeof(int)) != cudaSuccess ||
        cudaMemset(c->d_status, 0, sizeof(int)) != cudaSuccess || noalloc_preload() != RBFFD_OK) {
        cudaGetLastError();
        if (c->d_status) cudaFree(c->d_status);
        cudaStreamDestroy(c->stream);
        delete c;
        return RBFFD_ERR_CUDA;
    }
    *out = c;
    return RBFFD_OK;
}

int ctx_check_device_status(rbffd_ctx* ctx)
{
    int st = 0;
    RBFFD_CUDA_TRY(ctx, cudaMemcpyAsync(&st, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    RBFFD_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    if (st == DEV_STATUS_OK) return RBFFD_OK;
    RBFFD_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_status, 0, sizeof(int), ctx->stream));
    RBFFD_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return set_error(ctx, RBFFD_ERR_TIMEOUT, "a stage kernel gave up waiting for its bulk copies (device status %d)", st);
}

extern "C" int rbffd_ctx_destroy(rbffd_ctx* ctx)
{
    if (!ctx) return RBFFD_ERR_INVALID;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    grid_launches_forget(ctx);
    cudaStreamDestroy(ctx->stream);
    if (ctx->d_status) cudaFree(ctx->d_status);
    for (int* p : ctx->wait_pages) cudaFreeHost(p);
    keep_free(ctx, &ctx->stage);
    delete ctx;
    return RBFFD_OK;
}

extern "C" const char* rbffd_ctx_last_error(const rbffd_ctx* ctx) { return ctx ? ctx->last_error.c_str() : "null context"; }

extern "C" int rbffd_ctx_synchronize(rbffd_ctx* ctx)
{
    if (!ctx) return RBFFD_ERR_INVALID;
    RBFFD_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    bool gave_up = false;
    {
        std::lock_guard<std::mutex> lk(ctx->mu);
        for (const int* p : ctx->wait_pages)
            for (int k = 0; k < WAIT_PAGE; k++) gave_up |= ((const volatile int*)p)[k] != DEV_STATUS_OK;
    }
    if (gave_up)
        return set_error(ctx, RBFFD_ERR_TIMEOUT, "an advance gave up waiting: its PDE's state has to be set again");
    return RBFFD_OK;
}

int* ctx_wait_slot(rbffd_ctx* ctx)
{
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (ctx->wait_free.empty()) {
        int* p = nullptr;
        if (cudaHostAlloc((void**)&p, WAIT_PAGE * sizeof(int), cudaHostAllocMapped) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        memset(p, 0, WAIT_PAGE * sizeof(int));
        ctx->wait_pages.push_back(p);
        for (int k = WAIT_PAGE - 1; k >= 0; k--) ctx->wait_free.push_back(p + k);
    }
    int* s = ctx->wait_free.back();
    ctx->wait_free.pop_back();
    return s;
}

void ctx_wait_release(rbffd_ctx* ctx, int* slot)
{
    if (!slot) return;
    std::lock_guard<std::mutex> lk(ctx->mu);
    *(volatile int*)slot = DEV_STATUS_OK;
    ctx->wait_free.push_back(slot);
}

extern "C" int rbffd_ctx_mem_info(rbffd_ctx* ctx, size_t* held, size_t* free_bytes, size_t* total_bytes)
{
    if (!ctx) return RBFFD_ERR_INVALID;
    cudaSetDevice(ctx->device);
    size_t f = 0, t = 0;
    RBFFD_CUDA_TRY(ctx, cudaMemGetInfo(&f, &t));
    if (held) *held = ctx_in_use(ctx);
    if (free_bytes) *free_bytes = f;
    if (total_bytes) *total_bytes = t;
    return RBFFD_OK;
}

extern "C" int rbffd_ctx_stream(rbffd_ctx* ctx, void** stream)
{
    if (!ctx || !stream) return RBFFD_ERR_INVALID;
    *stream = (void*)ctx->stream;
    return RBFFD_OK;
}

// ---------------------------------------------------------------------------
// grid

// Host stencils [N][n_pad] (valid prefix len[i]) -> sliced ELL with centre padding.
__global__ void k_pack_stencils(const int* __restrict__ st_rm, const int* __restrict__ len, int N, int n_pad, int n4,
                                int nc, int* __restrict__ idx)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    int L = len[i];
    for (int s = 0; s < n4; s++) idx[sell_elem(i, s, nc)] = (s < L) ? st_rm[(size_t)i * n_pad + s] : i;
}

__global__ void k_xyz4(const double* __restrict__ xyz, int N, double4* __restrict__ out)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    out[i] = make_double4(xyz[3 * (size_t)i], xyz[3 * (size_t)i + 1], xyz[3 * (size_t)i + 2], 0.0);
}

extern "C" int rbffd_grid_create(rbffd_ctx* ctx, int N, const double* xyz, int n_pad, const int* st, const int* st_len,
                                 rbffd_grid** out)
{
    return rbffd_grid_create_ordered(ctx, N, xyz, n_pad, st, st_len, RBFFD_ORDER_MORTON, out);
}

extern "C" int rbffd_grid_create_ordered(rbffd_ctx* ctx, int N, const double* xyz, int n_pad, const int* st,
                                         const int* st_len, int order_method, rbffd_grid** out)
{
    if (!ctx || !out || !xyz || !st || N <= 0 || n_pad <= 0 || n_pad > 1024) return RBFFD_ERR_INVALID;
    *out = nullptr;
    // Host-side validation: every index in range, centre first, lengths in [1, n_pad].
    std::vector<int> len(N);
    for (int i = 0; i < N; i++) {
        int L = st_len ? st_len[i] : n_pad;
        if (L < 1 || L > n_pad)
            return set_error(ctx, RBFFD_ERR_INVALID, "stencil %d: length %d outside [1, %d]", i, L, n_pad);
        const int* row = st + (size_t)i * n_pad;
        if (row[0] != i)
            return set_error(ctx, RBFFD_ERR_INVALID,
                             "stencil %d: centre must be the first entry (found %d; rbffd.cpp:916-928)", i, row[0]);
        for (int s = 0; s < L; s++)
            if (row[s] < 0 || row[s] >= N)
                return set_error(ctx, RBFFD_ERR_INVALID, "stencil %d slot %d: node index %d outside [0, %d)", i, s,
                                 row[s], N);
        len[i] = L;
    }
    cudaSetDevice(ctx->device);
    rbffd_grid* g = new (std::nothrow) rbffd_grid();
    if (!g) return RBFFD_ERR_OOM;
    g->ctx = ctx;
    g->N = N;
    g->n_pad = n_pad;
    g->n4 = round_up(n_pad, 4);
    g->nc = g->n4 / 4;
    g->N32 = round_up(N, 32);
    // Internal order (rbffd_node_order): by default nodes along a 3-D Morton
    // curve, so consecutive rows are spatial neighbours and share most of the
    // nodes their stencils gather.
    g->h_perm.resize(N);
    g->h_iperm.resize(N);
    {
        const int rc = rbffd_node_order(N, xyz, n_pad, st, st_len, order_method, g->h_perm.data());
        if (rc) {
            delete g;
            return set_error(ctx, rc, "node order %d", order_method);
        }
        for (int i = 0; i < N; i++) g->h_iperm[g->h_perm[i]] = i;
    }
    std::vector<int> st_int((size_t)N * n_pad, 0);
    std::vector<double> xyz_int((size_t)N * 3);
    g->h_len.resize(N);
    for (int i = 0; i < N; i++) {
        const int o = g->h_perm[i];
        g->h_len[i] = len[o];
        for (int s = 0; s < len[o]; s++) st_int[(size_t)i * n_pad + s] = g->h_iperm[st[(size_t)o * n_pad + s]];
        for (int a = 0; a < 3; a++) xyz_int[3 * (size_t)i + a] = xyz[3 * (size_t)o + a];
    }
    size_t b_idx = (size_t)g->N32 * g->n4 * sizeof(int), b_len = (size_t)N * sizeof(int),
           b_xyz = (size_t)N * sizeof(double4);
    int rc;
    int* d_st = nullptr;
    double* d_x3 = nullptr;
    if ((rc = dev_alloc(ctx, (void**)&g->d_idx, b_idx)) || (rc = dev_alloc(ctx, (void**)&g->d_len, b_len)) ||
        (rc = dev_alloc(ctx, (void**)&g->d_xyz, b_xyz)) || (rc = dev_alloc(ctx, (void**)&g->d_perm, b_len)) ||
        (rc = dev_alloc(ctx, (void**)&d_st, (size_t)N * n_pad * sizeof(int))) ||
        (rc = dev_alloc(ctx, (void**)&d_x3, (size_t)N * 3 * sizeof(double)))) {
        dev_free(ctx, d_st, (size_t)N * n_pad * sizeof(int));
        dev_free(ctx, d_x3, (size_t)N * 3 * sizeof(double));
        rbffd_grid_destroy(g);
        return rc;
    }
    g->bytes = b_idx + 2 * b_len + b_xyz;
    cudaStream_t s = ctx->stream;
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess) e = cudaMemsetAsync(g->d_idx, 0, b_idx, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_st, st_int.data(), (size_t)N * n_pad * sizeof(int), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(g->d_len, g->h_len.data(), b_len, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(g->d_perm, g->h_perm.data(), b_len, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_x3, xyz_int.data(), (size_t)N * 3 * sizeof(double), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        int B = 256, G = (N + B - 1) / B;
        k_pack_stencils<<<G, B, 0, s>>>(d_st, g->d_len, N, n_pad, g->n4, g->nc, g->d_idx);
        k_xyz4<<<G, B, 0, s>>>(d_x3, N, g->d_xyz);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    dev_free(ctx, d_st, (size_t)N * n_pad * sizeof(int));
    dev_free(ctx, d_x3, (size_t)N * 3 * sizeof(double));
    if (e != cudaSuccess) {
        rbffd_grid_destroy(g);
        return cuda_error(ctx, e, "rbffd_grid_create");
    }
    *out = g;
    return RBFFD_OK;
}

static void halo_free(rbffd_grid* g, Halo* h)
{
    rbffd_ctx* ctx = g->ctx;
    if (h->d_whole) {  // grid_halo_whole: every array in one allocation
        dev_free(ctx, h->d_whole, h->b_whole);
        delete h;
        return;
    }
    dev_free(ctx, h->d_ptr, (size_t)(h->nblocks + 1) * sizeof(int));
    dev_free(ctx, h->d_rows, (size_t)(h->nblocks + 1) * sizeof(int));
    dev_free(ctx, h->d_nodes, h->b_nodes);
    dev_free(ctx, h->d_lidx, h->b_lidx);
    for (int k = 0; k < 4; k++) {
        dev_free(ctx, h->d_lidx_s[k], h->b_lidx);
        dev_free(ctx, h->d_slot_s[k], h->b_lidx);
    }
    delete h;
}

extern "C" int rbffd_grid_destroy(rbffd_grid* g)
{
    if (!g) return RBFFD_ERR_INVALID;
    rbffd_ctx* ctx = g->ctx;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    weights_work_free(g);
    size_t wsz = (size_t)g->N32 * g->n4;
    for (int t = 0; t < 16; t++) {
        dev_free(ctx, g->d_w64[t], wsz * sizeof(double));
        dev_free(ctx, g->d_w32[t], wsz * sizeof(float));
        dev_free(ctx, g->d_w32s[t], wsz * sizeof(float));
    }
    dev_free(ctx, g->d_idx, wsz * sizeof(int));
    dev_free(ctx, g->d_len, (size_t)g->N * sizeof(int));
    dev_free(ctx, g->d_perm, (size_t)g->N * sizeof(int));
    dev_free(ctx, g->d_xyz, (size_t)g->N * sizeof(double4));
    resident_free(g);
    for (auto& kv : g->halos) halo_free(g, kv.second);
    if (g->whole) halo_free(g, g->whole);
    for (Kept& f : g->field) keep_free(ctx, &f);
    keep_free(ctx, &g->idx_caller);
    delete g;
    return RBFFD_OK;
}

// Row blocks and their halos (see struct Halo).  Built on the host from the
// device's stencil array the first time a block size is used.
// Weights in a slot schedule: element e of the sliced ELL array (row i,
// scheduled slot t) takes row i's weight at its original slot slot[e], or 0
// for a padding entry.
__global__ void k_schedule_f32(const float* __restrict__ w, const unsigned short* __restrict__ slot, size_t n, int nc,
                               float* __restrict__ ws)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const size_t q = e >> 2;                      // (slice, chunk, lane) of the element
    const int i = (int)((q / 32) / nc) * 32 + (int)(q % 32);
    const unsigned short s = slot[e];
    ws[e] = s == SLOT_FREE ? 0.0f : w[sell_elem(i, s, nc)];
}

static void parallel_for(int count, const std::function<void(int)>& f)
{
    std::atomic<int> next(0);
    unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    std::vector<std::thread> pool;
    for (unsigned t = 0; t < hw; t++)
        pool.emplace_back([&]() {
            for (int k; (k = next.fetch_add(1)) < count;) f(k);
        });
    for (auto& t : pool) t.join();
}

// Slot schedule of one wavefront group (rows q0 .. q1-1, at most P) of a
// block whose halo has hn positions.  A row's reads of one step are 16-byte
// vectors of a 128/P-byte node record; the group's rows read in one
// shared-memory wavefront when their positions are different mod P (the bank
// group).  Each step is a maximum matching of rows to bank groups (Kuhn's
// augmenting paths): a row may take a remaining slot of that group
// (preferring the group it has most slots left in) or, while it has padding
// entries to spend, a padding entry placed in any free group.  Rows that stay
// unmatched take a remaining slot anyway (a conflict).
static void schedule_group(const rbffd_grid* g, const std::vector<unsigned short>& lidx, int q0, int q1, int hn,
                           int P, std::vector<unsigned short>& lidx_s, std::vector<unsigned short>& slot_s)
{
    const int nc = g->nc, n4 = g->n4, G = q1 - q0;
    std::vector<int> by[8][8];  // by[row][group]: remaining slots, the lowest last
    int realrem[8] = {}, freerem[8] = {};
    for (int r = 0; r < G; r++) {
        const int len = g->h_len[q0 + r];
        for (int s = len - 1; s >= 0; s--) by[r][lidx[sell_elem(q0 + r, s, nc)] & (P - 1)].push_back(s);
        realrem[r] = len;
        freerem[r] = n4 - len;
    }
    for (int t = 0; t < n4; t++) {
        int pref[8][8], npref[8] = {};
        for (int r = 0; r < G; r++) {
            int cs[8], k = 0;
            for (int c = 0; c < P; c++)
                if (!by[r][c].empty()) cs[k++] = c;
            std::sort(cs, cs + k, [&](int a, int b) { return by[r][a].size() > by[r][b].size(); });
            for (int j = 0; j < k; j++) pref[r][npref[r]++] = cs[j];
            if (freerem[r] > 0)
                for (int c = 0; c < P; c++)
                    if (by[r][c].empty()) pref[r][npref[r]++] = c;
        }
        int order[8];
        for (int r = 0; r < G; r++) order[r] = r;
        std::sort(order, order + G, [&](int a, int b) {
            if ((freerem[a] == 0) != (freerem[b] == 0)) return freerem[a] == 0;
            return npref[a] < npref[b];
        });
        int owner[8];
        for (int c = 0; c < P; c++) owner[c] = -1;
        std::function<bool(int, unsigned&)> augment = [&](int r, unsigned& seen) {
            for (int j = 0; j < npref[r]; j++) {
                const int c = pref[r][j];
                if (seen & (1u << c)) continue;
                seen |= 1u << c;
                if (owner[c] < 0 || augment(owner[c], seen)) {
                    owner[c] = r;
                    return true;
                }
            }
            return false;
        };
        for (int j = 0; j < G; j++) {
            unsigned seen = 0;
            augment(order[j], seen);
        }
        int colour[8];
        for (int r = 0; r < G; r++) colour[r] = -1;
        for (int c = 0; c < P; c++)
            if (owner[c] >= 0) colour[owner[c]] = c;
        for (int r = 0; r < G; r++) {
            const size_t e = sell_elem(q0 + r, t, nc);
            int c = colour[r];
            if (c < 0 || (by[r][c].empty() && freerem[r] == 0)) {  // unmatched: a conflicting slot
                c = -1;
                for (int k = 0; k < P; k++)
                    if (!by[r][k].empty() && (c < 0 || by[r][k].size() > by[r][c].size())) c = k;
            }
            if (c >= 0 && !by[r][c].empty()) {
                const int s = by[r][c].back();
                by[r][c].pop_back();
                realrem[r]--;
                slot_s[e] = (unsigned short)s;
                lidx_s[e] = lidx[sell_elem(q0 + r, s, nc)];
            } else {  // a padding entry, placed in group c (or 0)
                freerem[r]--;
                const int p = c < 0 ? 0 : c;
                slot_s[e] = SLOT_FREE;
                lidx_s[e] = (unsigned short)(p < hn ? p : p % std::max(hn, 1));
            }
        }
    }
}

int grid_halo_schedule(rbffd_grid* g, int R, int P, const Halo** out)
{
    rbffd_ctx* ctx = g->ctx;
    const int k = P == 2 ? 1 : (P == 4 ? 2 : (P == 8 ? 3 : -1));
    if (k < 0) return set_error(ctx, RBFFD_ERR_INVALID, "slot schedule for %d rows per wavefront", P);
    const Halo* hc = nullptr;
    int rc = grid_halo(g, R, &hc);
    if (rc) return rc;
    Halo* h = const_cast<Halo*>(hc);
    if (h->d_lidx_s[k]) {
        *out = h;
        return RBFFD_OK;
    }
    const size_t nidx = (size_t)g->N32 * g->n4;
    std::vector<unsigned short> lidx(nidx), lidx_s(nidx, 0), slot_s(nidx, SLOT_FREE);
    std::vector<int> rows(h->nblocks + 1), ptr(h->nblocks + 1);
    RBFFD_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    RBFFD_CUDA_TRY(ctx, cudaMemcpy(lidx.data(), h->d_lidx, nidx * sizeof(unsigned short), cudaMemcpyDeviceToHost));
    RBFFD_CUDA_TRY(ctx, cudaMemcpy(rows.data(), h->d_rows, rows.size() * sizeof(int), cudaMemcpyDeviceToHost));
    RBFFD_CUDA_TRY(ctx, cudaMemcpy(ptr.data(), h->d_ptr, ptr.size() * sizeof(int), cudaMemcpyDeviceToHost));
    parallel_for(h->nblocks, [&](int b) {
        const int hn = ptr[b + 1] - ptr[b];
        for (int q0 = rows[b]; q0 < rows[b + 1]; q0 += P)
            schedule_group(g, lidx, q0, std::min(rows[b + 1], q0 + P), hn, P, lidx_s, slot_s);
    });
    const size_t bytes = nidx * sizeof(unsigned short);
    if ((rc = dev_alloc(ctx, (void**)&h->d_lidx_s[k], bytes))) return rc;
    if ((rc = dev_alloc(ctx, (void**)&h->d_slot_s[k], bytes))) {
        dev_free(ctx, h->d_lidx_s[k], bytes);
        h->d_lidx_s[k] = nullptr;
        return rc;
    }
    cudaError_t e = cudaMemcpy(h->d_lidx_s[k], lidx_s.data(), bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(h->d_slot_s[k], slot_s.data(), bytes, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        dev_free(ctx, h->d_lidx_s[k], bytes);
        dev_free(ctx, h->d_slot_s[k], bytes);
        h->d_lidx_s[k] = h->d_slot_s[k] = nullptr;
        return cuda_error(ctx, e, "slot schedule upload");
    }
    g->bytes += 2 * bytes;
    *out = h;
    return RBFFD_OK;
}

int grid_halo(rbffd_grid* g, int R, const Halo** out)
{
    auto it = g->halos.find(R);
    if (it != g->halos.end()) {
        *out = it->second;
        return RBFFD_OK;
    }
    rbffd_ctx* ctx = g->ctx;
    if (R < 32 || R % 32) return set_error(ctx, RBFFD_ERR_INVALID, "rows per block %d must be a multiple of 32", R);
    const int N = g->N, nc = g->nc, n4 = g->n4;
    const size_t nidx = (size_t)g->N32 * n4;
    std::vector<int> idx(nidx);
    RBFFD_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    RBFFD_CUDA_TRY(ctx, cudaMemcpy(idx.data(), g->d_idx, nidx * sizeof(int), cudaMemcpyDeviceToHost));
    // Per-slice (32 rows) sorted unique node lists.
    const int nsl = (N + 31) / 32;
    std::vector<std::vector<int>> snodes(nsl);
    auto run = [&](int count, const std::function<void(int)>& f) {
        std::atomic<int> next(0);
        unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
        std::vector<std::thread> pool;
        for (unsigned t = 0; t < hw; t++)
            pool.emplace_back([&]() {
                for (int k; (k = next.fetch_add(1)) < count;) f(k);
            });
        for (auto& t : pool) t.join();
    };
    run(nsl, [&](int q) {
        std::vector<int>& v = snodes[q];
        for (int r = 32 * q; r < std::min(N, 32 * q + 32); r++)
            for (int s = 0; s < n4; s++) v.push_back(idx[sell_elem(r, s, nc)]);
        std::sort(v.begin(), v.end());
        v.erase(std::unique(v.begin(), v.end()), v.end());
    });
    auto merge = [](const std::vector<int>& x, const std::vector<int>& y) {
        std::vector<int> m;
        m.reserve(x.size() + y.size());
        std::set_union(x.begin(), x.end(), y.begin(), y.end(), std::back_inserter(m));
        return m;
    };
    // Cap on a block's halo: the 90th percentile of fixed R-row blocks' halos
    // (shared memory is sized by the largest halo, so outliers are split).
    const int spb = R / 32, nfixed = (nsl + spb - 1) / spb;
    std::vector<int> fsize(nfixed);
    run(nfixed, [&](int b) {
        std::vector<int> u;
        for (int q = b * spb; q < std::min(nsl, (b + 1) * spb); q++) u = merge(u, snodes[q]);
        fsize[b] = (int)u.size();
    });
    std::vector<int> sorted_f(fsize);
    std::sort(sorted_f.begin(), sorted_f.end());
    size_t cap = (size_t)sorted_f[(size_t)(0.9 * (sorted_f.size() - 1))];
    for (int q = 0; q < nsl; q++) cap = std::max(cap, snodes[q].size());
    if (cap > 65535) return set_error(ctx, RBFFD_ERR_UNSUPPORTED, "a block halo exceeds 65535 nodes");
    // Greedy partition: grow each block slice by slice while the halo stays under the cap.
    std::vector<int> bstart;
    std::vector<std::vector<int>> nodes;
    for (int q = 0; q < nsl;) {
        bstart.push_back(q);
        std::vector<int> cur = snodes[q++];
        while (q < nsl && q - bstart.back() < spb) {
            std::vector<int> m = merge(cur, snodes[q]);
            if (m.size() > cap) break;
            cur.swap(m);
            q++;
        }
        nodes.push_back(std::move(cur));
    }
    const int nblocks = (int)bstart.size();
    bstart.push_back(nsl);
    std::vector<int> rows(nblocks + 1);
    for (int b = 0; b <= nblocks; b++) rows[b] = std::min(N, 32 * bstart[b]);
    // Placement of each block's halo nodes in shared memory.  A block's kernel
    // reads, per stencil slot, one value (or 16-byte vector) per row; the 8
    // rows of a quarter-warp are served in one shared-memory wavefront only if
    // their nodes sit in different 16-byte bank groups (position mod 8).  A
    // greedy colouring gives the nodes read together different positions mod 8
    // where it can: position = 8 * rank + colour, padding slots repeat a node
    // of the block (staging stays branch-free).  Only positions change: the
    // arithmetic of every row is the same.
    std::vector<unsigned short> lidx(nidx, 0);
    std::vector<std::vector<int>> layout(nblocks);
    run(nblocks, [&](int b) {
        const std::vector<int>& v = nodes[b];
        const int K = (int)v.size(), r0 = rows[b], r1 = rows[b + 1];
        std::vector<int> kidx((size_t)(r1 - r0) * n4);  // sorted-halo index of each (row, slot)
        for (int r = r0; r < r1; r++)
            for (int s = 0; s < n4; s++)
                kidx[(size_t)(r - r0) * n4 + s] =
                    (int)(std::lower_bound(v.begin(), v.end(), idx[sell_elem(r, s, nc)]) - v.begin());
        // groups: the distinct nodes that 8 consecutive rows read at one slot
        std::vector<std::vector<int>> groups;
        std::vector<std::vector<int>> of_node(K);
        for (int q0 = r0; q0 < r1; q0 += 8)
            for (int s = 0; s < n4; s++) {
                std::vector<int> gset;
                for (int r = q0; r < std::min(r1, q0 + 8); r++) gset.push_back(kidx[(size_t)(r - r0) * n4 + s]);
                std::sort(gset.begin(), gset.end());
                gset.erase(std::unique(gset.begin(), gset.end()), gset.end());
                if (gset.size() < 2) continue;
                for (int k : gset) of_node[k].push_back((int)groups.size());
                groups.push_back(std::move(gset));
            }
        std::vector<int> order(K), colour(K, -1), used(8, 0);
        std::vector<std::array<int, 8>> cnt(groups.size());
        for (auto& c : cnt) c.fill(0);
        for (int k = 0; k < K; k++) order[k] = k;
        std::stable_sort(order.begin(), order.end(),
                         [&](int a, int c) { return of_node[a].size() > of_node[c].size(); });
        const int cap = (K + 7) / 8 + 1;
        for (int k : order) {
            int best = -1;
            long best_cost = 0;
            for (int c = 0; c < 8; c++) {
                if (used[c] >= cap) continue;
                long cost = 0;
                for (int g : of_node[k]) cost += cnt[g][c];
                if (best < 0 || cost < best_cost || (cost == best_cost && used[c] < used[best])) {
                    best = c;
                    best_cost = cost;
                }
            }
            colour[k] = best;
            used[best]++;
            for (int g : of_node[k]) cnt[g][best]++;
        }
        std::vector<int> pos(K), rank(8, 0);
        for (int k = 0; k < K; k++) pos[k] = 8 * rank[colour[k]]++ + colour[k];
        int hn = 0;
        for (int k = 0; k < K; k++) hn = std::max(hn, pos[k] + 1);
        std::vector<int>& lay = layout[b];
        lay.assign(hn, v[0]);
        for (int k = 0; k < K; k++) lay[pos[k]] = v[k];
        for (int r = r0; r < r1; r++)
            for (int s = 0; s < n4; s++)
                lidx[sell_elem(r, s, nc)] = (unsigned short)pos[kidx[(size_t)(r - r0) * n4 + s]];
    });
    std::vector<int> ptr(nblocks + 1, 0), flat;
    int max_halo = 0;
    for (int b = 0; b < nblocks; b++) {
        if (layout[b].size() > 65535) return set_error(ctx, RBFFD_ERR_UNSUPPORTED, "a block halo exceeds 65535 slots");
        ptr[b + 1] = ptr[b] + (int)layout[b].size();
        max_halo = std::max(max_halo, (int)layout[b].size());
    }
    flat.reserve(ptr[nblocks]);
    for (int b = 0; b < nblocks; b++) flat.insert(flat.end(), layout[b].begin(), layout[b].end());
    Halo* h = new (std::nothrow) Halo();
    if (!h) return RBFFD_ERR_OOM;
    h->R = R;
    h->nblocks = nblocks;
    h->max_halo = max_halo;
    const size_t b_ptr = ptr.size() * sizeof(int), b_nodes = flat.size() * sizeof(int),
                 b_lidx = nidx * sizeof(unsigned short);
    int rc;
    if ((rc = dev_alloc(ctx, (void**)&h->d_ptr, b_ptr)) || (rc = dev_alloc(ctx, (void**)&h->d_nodes, b_nodes)) ||
        (rc = dev_alloc(ctx, (void**)&h->d_lidx, b_lidx)) || (rc = dev_alloc(ctx, (void**)&h->d_rows, b_ptr))) {
        dev_free(ctx, h->d_ptr, b_ptr);
        dev_free(ctx, h->d_nodes, b_nodes);
        dev_free(ctx, h->d_lidx, b_lidx);
        delete h;
        return rc;
    }
    cudaError_t e = cudaMemcpy(h->d_ptr, ptr.data(), b_ptr, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(h->d_rows, rows.data(), b_ptr, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(h->d_nodes, flat.data(), b_nodes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(h->d_lidx, lidx.data(), b_lidx, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        dev_free(ctx, h->d_ptr, b_ptr);
        dev_free(ctx, h->d_nodes, b_nodes);
        dev_free(ctx, h->d_lidx, b_lidx);
        dev_free(ctx, h->d_rows, b_ptr);
        delete h;
        return cuda_error(ctx, e, "grid_halo upload");
    }
    h->b_nodes = b_nodes;
    h->b_lidx = b_lidx;
    g->bytes += 2 * b_ptr + b_nodes + b_lidx;
    g->halos[R] = h;
    *out = h;
    return RBFFD_OK;
}

// ---------------------------------------------------------------------------
// halos of whole blocks, built on the device (grid_halo_whole): one CTA per
// block of R rows marks the nodes its stencils read in a bitmap in shared
// memory; a node's halo position is its rank there (ascending node number, so
// consecutive rows' neighbours sit close together).  The host build above,
// whose positions avoid more bank conflicts, takes 20 ms at N = 40003, n = 37;
// this one 0.1 ms, and a device-resident stage is 3 to 8% slower for it: 10^5
// stages pay for the difference.

constexpr int WHOLE_THREADS = 512;
constexpr int WHOLE_MAX_BLOCKS = 256;
constexpr int WHOLE_ADJ = WHOLE_MAX_BLOCKS / 32;

// FILL = false: counts[b] = halo positions, adj[b] = bit per block read.
// FILL = true: nodes, lidx and the words read (rnode, rpos), each block's from
// its offsets; then the block's extra words (extra[eptr[b] ..]) at position pos_extra.
template <bool FILL>
__global__ void __launch_bounds__(WHOLE_THREADS) k_halo_whole(const int* __restrict__ idx, int N, int nc, int R, int words,
                                                              int* counts, unsigned* adj, const int* ptr, const int* rptr,
                                                              const int* eptr, const int* extra, int pos_extra, int* nodes,
                                                              unsigned short* lidx, int* rnode, unsigned short* rpos)
{
    extern __shared__ unsigned sh_whole[];
    unsigned* const bits = sh_whole;           // [words]
    int* const pre = (int*)(sh_whole + words); // [words] set bits before each word
    __shared__ int part[WHOLE_THREADS];
    __shared__ unsigned from[WHOLE_ADJ];
    const int b = blockIdx.x, tid = threadIdx.x;
    const int row0 = b * R, row1 = min(N, row0 + R), nrows = row1 - row0;
    for (int w = tid; w < words; w += WHOLE_THREADS) bits[w] = 0;
    if (tid < WHOLE_ADJ) from[tid] = 0;
    __syncthreads();
    for (int e = tid; e < nrows * nc; e += WHOLE_THREADS) {
        const int c = e / nrows, r = e - c * nrows;
        const int4 j = ld_idx4(idx + sell_off(row0 + r, c, nc));
        atomicOr(&bits[j.x >> 5], 1u << (j.x & 31));
        atomicOr(&bits[j.y >> 5], 1u << (j.y & 31));
        atomicOr(&bits[j.z >> 5], 1u << (j.z & 31));
        atomicOr(&bits[j.w >> 5], 1u << (j.w & 31));
    }
    __syncthreads();
    const int per = (words + WHOLE_THREADS - 1) / WHOLE_THREADS, w0 = min(words, tid * per), w1 = min(words, w0 + per);
    int sum = 0;
    for (int w = w0; w < w1; w++) sum += __popc(bits[w]);
    part[tid] = sum;
    __syncthreads();
    for (int o = 1; o < WHOLE_THREADS; o <<= 1) {  // inclusive sums
        const int v = tid >= o ? part[tid - o] : 0;
        __syncthreads();
        part[tid] += v;
        __syncthreads();
    }
    const int total = part[WHOLE_THREADS - 1];
    if (!FILL) {
        for (int w = w0; w < w1; w++)
            for (unsigned m = bits[w]; m; m &= m - 1) {
                const int o = (32 * w + __ffs(m) - 1) / R;
                if (o != b) atomicOr(&from[o >> 5], 1u << (o & 31));
            }
        __syncthreads();
        if (tid < WHOLE_ADJ) adj[b * WHOLE_ADJ + tid] = from[tid];
        if (tid == 0) counts[b] = total;
        return;
    }
    int at = part[tid] - sum;
    for (int w = w0; w < w1; w++) {
        pre[w] = at;
        for (unsigned m = bits[w]; m; m &= m - 1, at++) {
            const int j = 32 * w + __ffs(m) - 1;
            nodes[ptr[b] + at] = j;
            if (j < row0 || j >= row1) {  // every row of the block is in its halo (its own centre)
                const int k = rptr[b] + (j < row0 ? at : at - nrows);
                rnode[k] = j;
                rpos[k] = (unsigned short)at;
            }
        }
    }
    for (int e = tid; e < eptr[b + 1] - eptr[b]; e += WHOLE_THREADS) {
        const int k = rptr[b] + total - nrows + e;
        rnode[k] = extra[eptr[b] + e];
        rpos[k] = (unsigned short)pos_extra;
    }
    __syncthreads();
    auto rank = [&](int j) { return (unsigned short)(pre[j >> 5] + __popc(bits[j >> 5] & ((1u << (j & 31)) - 1))); };
    for (int e = tid; e < nrows * nc; e += WHOLE_THREADS) {
        const int c = e / nrows, r = e - c * nrows;
        const size_t o = sell_off(row0 + r, c, nc);
        const int4 j = ld_idx4(idx + o);
        *reinterpret_cast<ushort4*>(lidx + o) = make_ushort4(rank(j.x), rank(j.y), rank(j.z), rank(j.w));
    }
}

int grid_halo_whole_sizes(rbffd_grid* g, int R, int* max_halo, int* max_read)
{
    rbffd_ctx* ctx = g->ctx;
    const int N = g->N, nblocks = (N + R - 1) / R, words = (N + 31) / 32;
    const size_t smem = (size_t)words * 8;
    if (R < 32 || R % 32 || nblocks > WHOLE_MAX_BLOCKS || smem > 160 * 1024)
        return set_error(ctx, RBFFD_ERR_UNSUPPORTED, "whole halos of %d rows for %d nodes", R, N);
    if (g->whole_R != R) {
        cudaStream_t s = ctx->stream;
        int* d_cnt = nullptr;
        const size_t b_cnt = (size_t)nblocks * (1 + WHOLE_ADJ) * sizeof(int);
        std::vector<int> cnt((size_t)nblocks * (1 + WHOLE_ADJ));
        const int rc = dev_alloc(ctx, (void**)&d_cnt, b_cnt);
        if (rc) return rc;
        cudaError_t e =
            cudaFuncSetAttribute(k_halo_whole<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) {
            k_halo_whole<false><<<nblocks, WHOLE_THREADS, smem, s>>>(g->d_idx, N, g->nc, R, words, d_cnt,
                                                                     (unsigned*)(d_cnt + nblocks), nullptr, nullptr,
                                                                     nullptr, nullptr, 0, nullptr, nullptr, nullptr,
                                                                     nullptr);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(cnt.data(), d_cnt, b_cnt, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        dev_free(ctx, d_cnt, b_cnt);
        if (e != cudaSuccess) return cuda_error(ctx, e, "grid_halo_whole");
        // offsets, and the words that keep a block behind one that reads it without being read by it; uploaded
        // together: rows, ptr, rptr and eptr (nblocks + 1 each), then the extra words
        const unsigned* adj = (const unsigned*)(cnt.data() + nblocks);
        auto reads = [&](int b, int o) { return adj[b * WHOLE_ADJ + (o >> 5)] >> (o & 31) & 1; };
        const int nb1 = nblocks + 1;
        std::vector<int> meta(4 * (size_t)nb1, 0);
        int *const rows = meta.data(), *const ptr = rows + nb1, *const rptr = ptr + nb1, *const eptr = rptr + nb1;
        std::vector<int> extra;
        g->whole_max_halo = g->whole_max_read = 0;
        for (int b = 0; b < nblocks; b++) {
            rows[b] = b * R;
            const int nrows = std::min(N, (b + 1) * R) - b * R;
            for (int o = 0; o < nblocks; o++)
                if (o != b && reads(o, b) && !reads(b, o)) extra.push_back(o * R);
            eptr[b + 1] = (int)extra.size();
            ptr[b + 1] = ptr[b] + cnt[b];
            const int nread = cnt[b] - nrows + eptr[b + 1] - eptr[b];
            rptr[b + 1] = rptr[b] + nread;
            g->whole_max_halo = std::max(g->whole_max_halo, cnt[b]);
            g->whole_max_read = std::max(g->whole_max_read, nread);
        }
        rows[nblocks] = N;
        meta.insert(meta.end(), extra.begin(), extra.end());
        g->whole_refused = g->whole_max_halo > 65534;
        g->whole_meta = g->whole_refused ? std::vector<int>() : std::move(meta);
        g->whole_R = R;
        if (g->whole) {  // one block size at a time: the device's SM count fixes it
            cudaStreamSynchronize(s);
            g->bytes -= g->whole->b_whole;
            halo_free(g, g->whole);
            g->whole = nullptr;
        }
    }
    if (g->whole_refused) return set_error(ctx, RBFFD_ERR_UNSUPPORTED, "a block halo exceeds 65534 nodes");
    *max_halo = g->whole_max_halo;
    *max_read = g->whole_max_read;
    return RBFFD_OK;
}

int grid_halo_whole(rbffd_grid* g, int R, const Halo** out)
{
    rbffd_ctx* ctx = g->ctx;
    int max_halo = 0, max_read = 0;
    int rc = grid_halo_whole_sizes(g, R, &max_halo, &max_read);
    if (rc) return rc;
    if (g->whole) {
        *out = g->whole;
        return RBFFD_OK;
    }
    const int N = g->N, nblocks = (N + R - 1) / R, words = (N + 31) / 32, nb1 = nblocks + 1;
    const size_t smem = (size_t)words * 8;
    cudaStream_t s = ctx->stream;
    Halo* h = new (std::nothrow) Halo();
    if (!h) return RBFFD_ERR_OOM;
    h->R = R;
    h->nblocks = nblocks;
    h->max_halo = max_halo;
    h->max_read = max_read;
    h->nread = g->whole_meta[2 * nb1 + nblocks];
    const std::vector<int>& meta = g->whole_meta;
    const size_t nlidx = (size_t)g->N32 * g->n4, nhalo = (size_t)meta[nb1 + nblocks], nread = (size_t)meta[2 * nb1 + nblocks];
    // one allocation: lidx | rpos | rnode | nodes | meta (16-bit arrays of even length first)
    h->b_whole = (round_up((int)nread, 2) + nlidx) * sizeof(unsigned short) +
                 (nread + nhalo + meta.size()) * sizeof(int);
    if ((rc = dev_alloc(ctx, &h->d_whole, h->b_whole))) {
        delete h;
        return rc;
    }
    h->d_lidx = (unsigned short*)h->d_whole;
    h->d_rpos = h->d_lidx + nlidx;
    h->d_rnode = (int*)(h->d_rpos + round_up((int)nread, 2));
    h->d_nodes = h->d_rnode + nread;
    h->d_rows = h->d_nodes + nhalo;
    h->d_ptr = h->d_rows + nb1;
    h->d_rptr = h->d_ptr + nb1;
    cudaError_t e = cudaFuncSetAttribute(k_halo_whole<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(h->d_rows, meta.data(), meta.size() * sizeof(int), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        k_halo_whole<true><<<nblocks, WHOLE_THREADS, smem, s>>>(g->d_idx, N, g->nc, R, words, nullptr, nullptr, h->d_ptr,
                                                                h->d_rptr, h->d_rptr + nb1, h->d_rptr + 2 * nb1, max_halo,
                                                                h->d_nodes, h->d_lidx, h->d_rnode, h->d_rpos);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        halo_free(g, h);
        return cuda_error(ctx, e, "grid_halo_whole fill");
    }
    g->whole_meta = std::vector<int>();
    g->whole = h;
    g->bytes += h->b_whole;
    *out = h;
    return RBFFD_OK;
}

// ---------------------------------------------------------------------------
// caller order <-> internal order

template <typename E>
__global__ void k_permute(const E* __restrict__ src, E* __restrict__ dst, const int* __restrict__ perm, int N, int T,
                          int to_internal)
{
    size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)N * T) return;
    int i = (int)(e / T), t = (int)(e % T);
    size_t o = (size_t)perm[i] * T + t;
    if (to_internal)
        dst[e] = src[o];
    else
        dst[o] = src[e];
}

static int grid_permute(rbffd_grid* g, const void* src, void* dst, int T, int elem_bytes, cudaStream_t s, int to_int)
{
    size_t n = (size_t)g->N * T;
    int nb = (int)((n + 255) / 256);
    if (elem_bytes == 8)
        k_permute<unsigned long long><<<nb, 256, 0, s>>>((const unsigned long long*)src, (unsigned long long*)dst,
                                                         g->d_perm, g->N, T, to_int);
    else if (elem_bytes == 4)
        k_permute<unsigned int><<<nb, 256, 0, s>>>((const unsigned int*)src, (unsigned int*)dst, g->d_perm, g->N, T,
                                                   to_int);
    else
        return set_error(g->ctx, RBFFD_ERR_INVALID, "element size %d", elem_bytes);
    RBFFD_CUDA_TRY(g->ctx, cudaGetLastError());
    return RBFFD_OK;
}

int grid_to_internal(rbffd_grid* g, const void* src, void* dst, int T, int elem_bytes, cudaStream_t s)
{
    return grid_permute(g, src, dst, T, elem_bytes, s, 1);
}

int grid_to_caller(rbffd_grid* g, const void* src, void* dst, int T, int elem_bytes, cudaStream_t s)
{
    return grid_permute(g, src, dst, T, elem_bytes, s, 0);
}

int grid_permute_preload()
{
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, k_permute<unsigned long long>) != cudaSuccess ||
        cudaFuncGetAttributes(&a, k_permute<unsigned int>) != cudaSuccess)
        return RBFFD_ERR_CUDA;
    return RBFFD_OK;
}

extern "C" int rbffd_grid_nbytes(const rbffd_grid* g, size_t* bytes)
{
    if (!g || !bytes) return RBFFD_ERR_INVALID;
    std::lock_guard<std::mutex> lk(g->ctx->kept_mu);
    *bytes = g->bytes + g->idx_caller.bytes;
    for (const Kept& f : g->field) *bytes += f.bytes;
    return RBFFD_OK;
}

// ---------------------------------------------------------------------------
// weights in and out

// Rows [c0, c1) of the caller's host layout [N][n_pad] (w_rm: from row c0) <->
// sliced ELL in internal order (internal row i is the caller's row perm[i]), one
// thread per row and 4-slot chunk: whole 32-byte sectors on both sides.  Into
// the grid: zero beyond the stencil length.
__global__ void k_pad_rows(const double* __restrict__ w_rm, const int* __restrict__ len, const int* __restrict__ perm,
                           int N, int n_pad, int nc, int c0, int c1, double* __restrict__ w)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(e / 32 / nc) * 32 + (int)(e % 32), c = (int)(e / 32 % nc);
    if (i >= N) return;
    const int o = perm[i];
    if (o < c0 || o >= c1) return;
    const int L = len[i];
    const double* src = w_rm + (size_t)(o - c0) * n_pad + 4 * c;
    double* dst = w + sell_off(i, c, nc);
#pragma unroll
    for (int s = 0; s < 4; s++) dst[s] = 4 * c + s < L ? src[s] : 0.0;
}

__global__ void k_unpad_rows(const double* __restrict__ w, const int* __restrict__ perm, int N, int n_pad, int nc, int c0,
                             int c1, double* __restrict__ w_rm)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(e / 32 / nc) * 32 + (int)(e % 32), c = (int)(e / 32 % nc);
    if (i >= N) return;
    const int o = perm[i];
    if (o < c0 || o >= c1) return;
    double v[4];
    ld_w4(w + sell_off(i, c, nc), v);
    double* dst = w_rm + (size_t)(o - c0) * n_pad + 4 * c;
#pragma unroll
    for (int s = 0; s < 4; s++)
        if (4 * c + s < n_pad) dst[s] = v[s];
}

__global__ void k_cast_f32(const double* __restrict__ a, float* __restrict__ b, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) b[i] = __double2float_rn(a[i]);
}

int grid_make_f32(rbffd_grid* g, int op)
{
    rbffd_ctx* ctx = g->ctx;
    size_t n = (size_t)g->N32 * g->n4;
    if (!g->d_w32[op]) {
        int rc = dev_alloc(ctx, (void**)&g->d_w32[op], n * sizeof(float));
        if (rc) return rc;
        g->bytes += n * sizeof(float);
    }
    k_cast_f32<<<std::max(1, std::min<int>((int)((n + 255) / 256), ctx->sm_count * 16)), 256, 0, ctx->stream>>>(
        g->d_w64[op], g->d_w32[op], n);
    RBFFD_CUDA_TRY(ctx, cudaGetLastError());
    g->w32_ver[op]++;
    if (g->d_w32s[op]) {  // keep the scheduled copy in step
        const Halo* h = g->halos.at(g->sched_R);
        k_schedule_f32<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(g->d_w32[op], h->d_slot_s[3], n, g->nc,
                                                                          g->d_w32s[op]);
        RBFFD_CUDA_TRY(ctx, cudaGetLastError());
    }
    return RBFFD_OK;
}

int grid_schedule_weights(rbffd_grid* g, const float* src, const unsigned short* slot, float* dst, cudaStream_t s)
{
    const size_t n = (size_t)g->N32 * g->n4;
    k_schedule_f32<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, slot, n, g->nc, dst);
    RBFFD_CUDA_TRY(g->ctx, cudaGetLastError());
    return RBFFD_OK;
}

int grid_f32_scheduled(rbffd_grid* g, int R, int op, const float** out)
{
    rbffd_ctx* ctx = g->ctx;
    // the grid's scheduled copies (d_w32s) all follow the 8-row schedule of one halo
    if (g->sched_R != 0 && g->sched_R != R)
        return set_error(ctx, RBFFD_ERR_UNSUPPORTED, "a grid keeps its scheduled FP32 weights for one block size");
    const Halo* hs = nullptr;
    int rc = grid_halo_schedule(g, R, 8, &hs);
    if (rc) return rc;
    g->sched_R = R;
    if (!g->d_w32[op] && (rc = grid_make_f32(g, op))) return rc;
    if (!g->d_w32s[op]) {
        const size_t n = (size_t)g->N32 * g->n4;
        if ((rc = dev_alloc(ctx, (void**)&g->d_w32s[op], n * sizeof(float)))) return rc;
        g->bytes += n * sizeof(float);
        const Halo* h = g->halos.at(g->sched_R);
        k_schedule_f32<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(g->d_w32[op], h->d_slot_s[3], n, g->nc,
                                                                          g->d_w32s[op]);
        RBFFD_CUDA_TRY(ctx, cudaGetLastError());
    }
    *out = g->d_w32s[op];
    return RBFFD_OK;
}

// Allocate (once) the FP64 array of operator `op`.
int grid_alloc_w64(rbffd_grid* g, int op)
{
    if (g->d_w64[op]) return RBFFD_OK;
    size_t n = (size_t)g->N32 * g->n4;
    int rc = dev_alloc(g->ctx, (void**)&g->d_w64[op], n * sizeof(double));
    if (rc) return rc;
    g->bytes += n * sizeof(double);
    RBFFD_CUDA_TRY(g->ctx, cudaMemsetAsync(g->d_w64[op], 0, n * sizeof(double), g->ctx->stream));
    return RBFFD_OK;
}

// The context's staging buffer for weights on their way in or out, of the size
// asked for up to STAGE_MAX (larger moves go in parts), kept between calls (Kept).
// The caller holds ctx->stage_mu and has finished its use of the buffer when it
// lets go.  An allocation per call took longer than the move itself (0.3 ms at 1 MB).
constexpr size_t STAGE_MAX = (size_t)16 << 20;

// Move one operator's weights between the host layout and w64: in parts of whole rows.
static int weights_move(rbffd_grid* g, double* w64, const double* in, double* out)
{
    rbffd_ctx* ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    std::lock_guard<std::mutex> lk(ctx->stage_mu);
    const size_t row = (size_t)g->n_pad * sizeof(double);
    double* const stage = (double*)keep_take(ctx, &ctx->stage, std::min((size_t)g->N * row, STAGE_MAX));
    if (!stage) {
        keep_release(ctx, &ctx->stage);
        return RBFFD_ERR_OOM;
    }
    const int part = (int)std::min<size_t>((size_t)g->N, ctx->stage.bytes / row);
    const unsigned nb = (unsigned)(((size_t)g->N32 * g->nc + 255) / 256);
    cudaError_t e = cudaSuccess;
    for (int c0 = 0; e == cudaSuccess && c0 < g->N; c0 += part) {
        const int c1 = std::min(g->N, c0 + part);
        const size_t n = (size_t)(c1 - c0) * row;
        if (in) {
            e = cudaMemcpyAsync(stage, in + (size_t)c0 * g->n_pad, n, cudaMemcpyHostToDevice, s);
            if (e != cudaSuccess) break;
            k_pad_rows<<<nb, 256, 0, s>>>(stage, g->d_len, g->d_perm, g->N, g->n_pad, g->nc, c0, c1, w64);
            e = cudaGetLastError();
        } else {
            k_unpad_rows<<<nb, 256, 0, s>>>(w64, g->d_perm, g->N, g->n_pad, g->nc, c0, c1, stage);
            e = cudaGetLastError();
            if (e == cudaSuccess) e = cudaMemcpyAsync(out + (size_t)c0 * g->n_pad, stage, n, cudaMemcpyDeviceToHost, s);
        }
    }
    const cudaError_t f = cudaStreamSynchronize(s);
    keep_release(ctx, &ctx->stage);
    if (e == cudaSuccess) e = f;
    return e == cudaSuccess ? RBFFD_OK : cuda_error(ctx, e, in ? "rbffd_weights_set" : "rbffd_weights_get");
}

extern "C" int rbffd_weights_set(rbffd_grid* g, unsigned der_type, const double* w)
{
    if (!g || !w) return RBFFD_ERR_INVALID;
    int op = der_index(der_type);
    if (op < 0) return set_error(g->ctx, RBFFD_ERR_INVALID, "der_type 0x%x is not a single operator", der_type);
    rbffd_ctx* ctx = g->ctx;
    cudaSetDevice(ctx->device);
    int rc = grid_alloc_w64(g, op);
    if (rc) return rc;
    if ((rc = weights_move(g, g->d_w64[op], w, nullptr))) return rc;
    if ((rc = grid_make_f32(g, op))) return rc;
    RBFFD_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return RBFFD_OK;
}

extern "C" int rbffd_weights_get(rbffd_grid* g, unsigned der_type, double* w)
{
    if (!g || !w) return RBFFD_ERR_INVALID;
    int op = der_index(der_type);
    if (op < 0) return set_error(g->ctx, RBFFD_ERR_INVALID, "der_type 0x%x is not a single operator", der_type);
    if (!g->d_w64[op]) return set_error(g->ctx, RBFFD_ERR_STATE, "weights for der_type 0x%x not computed", der_type);
    cudaSetDevice(g->ctx->device);
    return weights_move(g, g->d_w64[op], nullptr, w);
}

// ---------------------------------------------------------------------------
// K2: ELL apply.  G lanes per (row, tracer); lane g handles the 4-slot chunks
// g, g+G, ...; partial sums combined by xor-shuffle.  With G == 1 the
// accumulation order is the reference's (s = 0 .. n-1, rbffd.cpp:680-684) and
// FP64 results equal those of a fused-multiply-add CPU loop.

// PLAIN: each multiply-add rounded twice, product then sum (madd, ell.cuh):
// the reference's own build, whose x86-64 flags have no FMA.
template <typename T, int G, bool PLAIN = false>
__global__ void __launch_bounds__(256) k_ell_apply(const int* __restrict__ idx, const T* __restrict__ w, int nc,
                                                   const T* __restrict__ u, T* __restrict__ out, int start, int count,
                                                   int T_tr)
{
    int gt = blockIdx.x * blockDim.x + threadIdx.x;
    int r = gt / G, lane = gt % G;
    int rows = count * T_tr;
    bool active = r < rows;
    int i = start + (active ? r / T_tr : 0), t = active ? r % T_tr : 0;
    T acc = T(0);
    if (active) {
        for (int c = lane; c < nc; c += G) {
            const size_t o = sell_off(i, c, nc);
            int4 j = ld_idx4(idx + o);
            T wv[4];
            ld_w4(w + o, wv);
            acc = madd<T, PLAIN>(wv[0], __ldg(u + (size_t)j.x * T_tr + t), acc);
            acc = madd<T, PLAIN>(wv[1], __ldg(u + (size_t)j.y * T_tr + t), acc);
            acc = madd<T, PLAIN>(wv[2], __ldg(u + (size_t)j.z * T_tr + t), acc);
            acc = madd<T, PLAIN>(wv[3], __ldg(u + (size_t)j.w * T_tr + t), acc);
        }
    }
    acc = group_sum<G>(acc);
    if (active && lane == 0) out[(size_t)i * T_tr + t] = acc;
}

template <typename T>
static void launch_apply(rbffd_grid* g, const T* w, const T* u, T* out, int start, int count, int T_tr, int G,
                         cudaStream_t s)
{
    long long threads = (long long)count * T_tr * G;
    int B = 256, nb = (int)((threads + B - 1) / B);
    switch (G) {
    case 1: k_ell_apply<T, 1><<<nb, B, 0, s>>>(g->d_idx, w, g->nc, u, out, start, count, T_tr); break;
    case 2: k_ell_apply<T, 2><<<nb, B, 0, s>>>(g->d_idx, w, g->nc, u, out, start, count, T_tr); break;
    case 4: k_ell_apply<T, 4><<<nb, B, 0, s>>>(g->d_idx, w, g->nc, u, out, start, count, T_tr); break;
    default: k_ell_apply<T, 8><<<nb, B, 0, s>>>(g->d_idx, w, g->nc, u, out, start, count, T_tr); break;
    }
}

// Used by the unfused RK4 path as well (rk4.cu).
int grid_apply_dev(rbffd_grid* g, int op, int dtype, int T_tr, const void* u, void* out, int start, int count, int G,
                   cudaStream_t s)
{
    if (dtype == RBFFD_F64) {
        if (!g->d_w64[op]) return set_error(g->ctx, RBFFD_ERR_STATE, "weights of operator bit %d not computed", op);
        launch_apply<double>(g, g->d_w64[op], (const double*)u, (double*)out, start, count, T_tr, G, s);
    } else {
        if (!g->d_w32[op]) return set_error(g->ctx, RBFFD_ERR_STATE, "weights of operator bit %d not computed", op);
        launch_apply<float>(g, g->d_w32[op], (const float*)u, (float*)out, start, count, T_tr, G, s);
    }
    RBFFD_CUDA_TRY(g->ctx, cudaGetLastError());
    return RBFFD_OK;
}

int grid_apply_dev_plain(rbffd_grid* g, int op, int T_tr, const double* u, double* out, int start, int count,
                         cudaStream_t s)
{
    if (!g->d_w64[op]) return set_error(g->ctx, RBFFD_ERR_STATE, "weights of operator bit %d not computed", op);
    long long threads = (long long)count * T_tr;
    int nb = (int)((threads + 255) / 256);
    k_ell_apply<double, 1, true><<<nb, 256, 0, s>>>(g->d_idx, g->d_w64[op], g->nc, u, out, start, count, T_tr);
    RBFFD_CUDA_TRY(g->ctx, cudaGetLastError());
    return RBFFD_OK;
}

// K2 in the caller's node order: one launch for a whole rbffd_apply(_dev) call.
// idx: the stencils with the caller's node numbers (grid_caller_index); or the
// grid's own, u reordered to match or, THROUGH, each taken through perm (internal
// node -> caller's node).  A row's sum is stored at the caller's node.  U: type of u and out (FP64 host fields of an FP32 call are
// rounded as they are read).  VEC: tracers per lane, one or a 16-byte vector;
// T_tr / VEC lanes of a row share its weights and indices.  Slots in stencil
// order, one lane per (row, vector): k_ell_apply's sums with G = 1.
//
// Bound by the gathers (L1) and, on small grids, by the latency of the dependent
// loads index -> value, so four chunks' loads are in flight for single values.
template <typename T, typename U, int VEC, bool PLAIN, bool THROUGH>
__global__ void __launch_bounds__(256) k_apply_caller(const int* __restrict__ idx, const T* __restrict__ w,
                                                      const int* __restrict__ perm, int nc, int N,
                                                      const U* __restrict__ u, U* __restrict__ out, int T_tr)
{
    const int lanes = T_tr / VEC;
    const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long row = gt / lanes;
    if (row >= N) return;
    const int i = (int)row, t = (int)(gt - row * lanes) * VEC;
    const U* const ut = u + t;
    T acc[VEC];
#pragma unroll
    for (int v = 0; v < VEC; v++) acc[v] = T(0);
#pragma unroll(VEC == 1 ? 4 : 2)
    for (int c = 0; c < nc; c++) {
        const size_t o = sell_off(i, c, nc);
        const int4 j4 = ld_idx4(idx + o);
        const int j[4] = {j4.x, j4.y, j4.z, j4.w};
        T wv[4];
        ld_w4(w + o, wv);
        U x[4][VEC];
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const U* const q = ut + (size_t)(THROUGH ? __ldg(perm + j[s]) : j[s]) * T_tr;
            if constexpr (VEC == 1) {
                x[s][0] = __ldg(q);
            } else if constexpr (sizeof(U) == 4) {
                const float4 z = __ldg(reinterpret_cast<const float4*>(q));
                memcpy(x[s], &z, sizeof z);
            } else {
                const double2 z = __ldg(reinterpret_cast<const double2*>(q));
                memcpy(x[s], &z, sizeof z);
            }
        }
#pragma unroll
        for (int s = 0; s < 4; s++)
#pragma unroll
            for (int v = 0; v < VEC; v++) acc[v] = madd<T, PLAIN>(wv[s], (T)x[s][v], acc[v]);
    }
    U* const q = out + (size_t)perm[i] * T_tr + t;
#pragma unroll
    for (int v = 0; v < VEC; v++) q[v] = (U)acc[v];
}

// Threads per block: 256, fewer while that leaves SMs without a block.
static int apply_block(const rbffd_ctx* ctx, long long threads)
{
    const long long per_sm = threads / std::max(1, ctx->sm_count);
    return (int)std::min<long long>(256, std::max<long long>(32, per_sm / 32 * 32));
}

__global__ void k_caller_index(const int4* __restrict__ idx, const int* __restrict__ perm, size_t n, int4* __restrict__ out)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const int4 j = idx[e];
    out[e] = make_int4(perm[j.x], perm[j.y], perm[j.z], perm[j.w]);
}

// The stencils with the caller's node numbers, made at a grid's 16th application
// to wide records: a look-up through perm per slot instead takes 137 against 108
// us a call at N = 163842, n = 101 with 16 FP32 tracers, the allocation 1.7 ms.
// nullptr before that, and if there is no memory for them.
static const int* grid_caller_index(rbffd_grid* g)
{
    const size_t n = (size_t)g->N32 * g->n4;
    {
        std::lock_guard<std::mutex> lk(g->ctx->kept_mu);
        if (g->idx_caller.p) {
            g->idx_caller.busy = true;
            return (const int*)g->idx_caller.p;
        }
    }
    if (g->wide_applies == 16) g->wide_applies = 0;  // not had, or given back: asked for again later
    if (++g->wide_applies < 16) return nullptr;
    KeepError keep(g->ctx);
    int* const p = (int*)keep_take(g->ctx, &g->idx_caller, n * sizeof(int));
    if (p)
        k_caller_index<<<(unsigned)((n / 4 + 255) / 256), 256, 0, g->ctx->stream>>>((const int4*)g->d_idx, g->d_perm,
                                                                                   n / 4, (int4*)p);
    return p;
}

template <typename T, typename U, bool PLAIN, bool THROUGH>
static void launch_apply_caller_t(rbffd_grid* g, const int* idx, const T* w, const U* u, U* out, int T_tr, cudaStream_t s)
{
    constexpr int V = 16 / (int)sizeof(U);
    const bool vec = T_tr % V == 0 && (((uintptr_t)u | (uintptr_t)out) & 15) == 0;
    const long long threads = (long long)g->N * (vec ? T_tr / V : T_tr);
    const int B = apply_block(g->ctx, threads);
    const unsigned nb = (unsigned)((threads + B - 1) / B);
    if (vec)
        k_apply_caller<T, U, V, PLAIN, THROUGH><<<nb, B, 0, s>>>(idx, w, g->d_perm, g->nc, g->N, u, out, T_tr);
    else
        k_apply_caller<T, U, 1, PLAIN, THROUGH><<<nb, B, 0, s>>>(idx, w, g->d_perm, g->nc, g->N, u, out, T_tr);
}

// Fields of N doubles kept with the grid: 0 and 1 rbffd_apply's field and
// derivative, 2 a reordered field (2 N; separate, so that the first calls on
// grids up to 65536 nodes stay with small allocations); nullptr without memory.
static double* grid_field(rbffd_grid* g, int k)
{
    return (double*)keep_take(g->ctx, &g->field[k], (k < 2 ? 1 : 2) * (size_t)g->N * sizeof(double));
}

// A call's use of the grid's kept buffers, one call at a time; it ends with the call's work done.
struct ApplyUse {
    rbffd_grid* g;
    std::lock_guard<std::mutex> lk;
    explicit ApplyUse(rbffd_grid* q) : g(q), lk(q->apply_mu) {}
    ~ApplyUse()
    {
        std::lock_guard<std::mutex> l2(g->ctx->kept_mu);
        for (Kept& f : g->field) f.busy = false;
        g->idx_caller.busy = false;
    }
};

// Node records of at most half a 32-byte sector: on grids past 65536 nodes the
// field is reordered first, since the caller's order spreads a row's neighbours
// over a sector each, four times the L1 that the internal order takes (35 us
// against 3 + 17 us at N = 163842, n = 50, FP64, one tracer); below, the numbers
// go through perm (at N = 40962 10.5 against 2.3 + 7.4 us and a launch more).
// Wider records are gathered from the caller's order.
template <typename T, typename U, bool PLAIN>
static void launch_apply_caller(rbffd_grid* g, const T* w, const U* u, U* out, int T_tr, cudaStream_t s)
{
    const int* idx = nullptr;
    if (T_tr * sizeof(U) > 16) {
        idx = grid_caller_index(g);
    } else if (g->N > 65536) {
        KeepError keep(g->ctx);
        U* const ui = (U*)grid_field(g, 2);
        if (ui && grid_to_internal(g, u, ui, T_tr, sizeof(U), s) == RBFFD_OK) {
            idx = g->d_idx;
            u = ui;
        }
    }
    if (idx)
        launch_apply_caller_t<T, U, PLAIN, false>(g, idx, w, u, out, T_tr, s);
    else
        launch_apply_caller_t<T, U, PLAIN, true>(g, g->d_idx, w, u, out, T_tr, s);
}

// deriv = the operator's weights on u, device fields in the caller's order, on the context's stream.
static void apply_caller(rbffd_grid* g, int op, int dtype, int T_tr, const void* u, void* out, bool doubles, cudaStream_t s)
{
    if (dtype == RBFFD_F64 && g->ctx->arith == RBFFD_ARITH_UNFUSED)
        launch_apply_caller<double, double, true>(g, g->d_w64[op], (const double*)u, (double*)out, T_tr, s);
    else if (dtype == RBFFD_F64)
        launch_apply_caller<double, double, false>(g, g->d_w64[op], (const double*)u, (double*)out, T_tr, s);
    else if (doubles)
        launch_apply_caller<float, double, false>(g, g->d_w32[op], (const double*)u, (double*)out, T_tr, s);
    else
        launch_apply_caller<float, float, false>(g, g->d_w32[op], (const float*)u, (float*)out, T_tr, s);
}

extern "C" int rbffd_ctx_set_arithmetic(rbffd_ctx* ctx, int arith)
{
    if (!ctx) return RBFFD_ERR_INVALID;
    if (arith != RBFFD_ARITH_FUSED && arith != RBFFD_ARITH_UNFUSED)
        return set_error(ctx, RBFFD_ERR_INVALID, "unknown arithmetic %d", arith);
    ctx->arith = arith;
    return RBFFD_OK;
}

extern "C" int rbffd_ctx_get_arithmetic(rbffd_ctx* ctx, int* arith)
{
    if (!ctx || !arith) return RBFFD_ERR_INVALID;
    *arith = ctx->arith;
    return RBFFD_OK;
}

extern "C" int rbffd_apply(rbffd_grid* g, unsigned der_type, int dtype, unsigned start, unsigned count, const double* u,
                           double* deriv)
{
    if (!g || !u || !deriv) return RBFFD_ERR_INVALID;
    if (dtype != RBFFD_F32 && dtype != RBFFD_F64) return set_error(g->ctx, RBFFD_ERR_INVALID, "bad dtype %d", dtype);
    if ((size_t)start + count > (size_t)g->N) return set_error(g->ctx, RBFFD_ERR_INVALID, "range outside the grid");
    int op = der_index(der_type);
    if (op < 0) return set_error(g->ctx, RBFFD_ERR_INVALID, "der_type 0x%x is not a single operator", der_type);
    if (count == 0) return RBFFD_OK;
    rbffd_ctx* ctx = g->ctx;
    cudaSetDevice(ctx->device);
    int N = g->N;
    ApplyUse use(g);
    // the field and its derivative on the device, in the caller's order; kept with the grid
    const size_t b64 = (size_t)N * sizeof(double);
    double *const du = grid_field(g, 0), *const dd = grid_field(g, 1);
    if (!du || !dd) return RBFFD_ERR_OOM;
    cudaStream_t s = ctx->stream;
    if (!(dtype == RBFFD_F64 ? (const void*)g->d_w64[op] : (const void*)g->d_w32[op]))
        return set_error(ctx, RBFFD_ERR_STATE, "weights of operator bit %d not computed", op);
    cudaError_t e = cudaMemcpyAsync(du, u, b64, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        apply_caller(g, op, dtype, 1, du, dd, true, s);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(deriv + start, dd + start, (size_t)count * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(ctx, e, "rbffd_apply");
    return RBFFD_OK;
}

extern "C" int rbffd_apply_dev(rbffd_grid* g, unsigned der_type, int dtype, int ntracers, const void* u_dev,
                               void* deriv_dev)
{
    if (!g || !u_dev || !deriv_dev || ntracers < 1) return RBFFD_ERR_INVALID;
    if (dtype != RBFFD_F32 && dtype != RBFFD_F64) return set_error(g->ctx, RBFFD_ERR_INVALID, "bad dtype %d", dtype);
    int op = der_index(der_type);
    if (op < 0) return set_error(g->ctx, RBFFD_ERR_INVALID, "der_type 0x%x is not a single operator", der_type);
    rbffd_ctx* ctx = g->ctx;
    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    if (!(dtype == RBFFD_F64 ? (const void*)g->d_w64[op] : (const void*)g->d_w32[op]))
        return set_error(ctx, RBFFD_ERR_STATE, "weights of operator bit %d not computed", op);
    ApplyUse use(g);
    // a result written over the field (or part of it): from a copy
    const size_t bytes = (size_t)g->N * ntracers * (dtype == RBFFD_F64 ? 8 : 4);
    void* copy = nullptr;
    const char *ub = (const char*)u_dev, *db = (const char*)deriv_dev;
    if (ub < db + bytes && db < ub + bytes) {
        const int rc = dev_alloc(ctx, &copy, bytes);
        if (rc) return rc;
        const cudaError_t e = cudaMemcpyAsync(copy, u_dev, bytes, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) {
            dev_free(ctx, copy, bytes);
            return cuda_error(ctx, e, "rbffd_apply_dev copy");
        }
        u_dev = copy;
    }
    apply_caller(g, op, dtype, ntracers, u_dev, deriv_dev, false, s);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    dev_free(ctx, copy, bytes);
    if (e != cudaSuccess) return cuda_error(ctx, e, "rbffd_apply_dev");
    return RBFFD_OK;
}
