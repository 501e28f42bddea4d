// sparse.cu -- CSR containers, row canonicalisation, transpose, scans,
// deterministic reductions and the FP64 SpMV primitives of the C ABI.
#include <cub/cub.cuh>

#include <atomic>
#include <climits>
#include <mutex>
#include <unordered_map>

#include "handle_heap.cuh"
#include "rb_internal.cuh"
#include "spmv.cuh"

namespace rb {

// ------------------------------------------------------------- context --
namespace {
cudaStream_t g_stream = nullptr;
cudaStream_t g_own_stream = nullptr;
int g_sms = 0;
thread_local std::string g_last_error;
}  // namespace

void set_last_error(const std::string& msg) { g_last_error = msg; }

long long& launch_counter() {
    static long long c = 0;
    return c;
}
long long& device_alloc_counter() {
    static long long c = 0;
    return c;
}
const char* last_error_cstr() { return g_last_error.c_str(); }

static cudaStream_t own_stream() {
    if (!g_own_stream) RB_CUDA(cudaStreamCreateWithFlags(&g_own_stream, cudaStreamNonBlocking));
    return g_own_stream;
}

cudaStream_t stream() {
    if (!g_stream) g_stream = own_stream();
    return g_stream;
}

void set_stream(cudaStream_t s) { g_stream = s ? s : nullptr; }

// ------------------------------------------------------- device memory --
// A setup makes about 500 allocations.  With cudaMalloc and cudaFree (which
// also waits for the device) they were most of its time; from a
// stream-ordered pool they cost the host a microsecond or two each and the
// device nothing (64^3 27-point setup 62.9 -> 25.7 ms, 256^2 forward and
// adjoint solve 37.0 -> 14.0 ms).  The pool keeps at most kPoolKeep bytes
// of freed memory: the driver gives back what is above at every
// synchronisation, and an allocation that fails gives back the rest and
// tries once more; once the last array is freed all but kIdleKeep goes back,
// and rb_trim gives back whatever is not in use (not all of it at once: a
// differentiated solve makes and frees all its handles in every step, 37 ms
// with nothing kept).  Arrays of kPoolLargest and more stay with cudaMalloc:
// pooled, the gigabytes a large hierarchy frees are unmapped at the next
// synchronisation, wherever it falls (a 192^3 setup 700 -> 1720 ms and the
// first solve after it 10.8 -> 380 ms; with the limit 606 ms and as before).
namespace {
constexpr unsigned long long kPoolKeep = 2ull << 30;
constexpr size_t kPoolLargest = (size_t)64 << 20;
constexpr size_t kIdleKeep = (size_t)256 << 20;     // of the pool with no array left
constexpr size_t kIdleSlabs = (size_t)128 << 20;    // of the handles' slabs then
constexpr int kMaxDevices = 64;
std::mutex g_pool_mu;
cudaMemPool_t g_pools[kMaxDevices] = {};
thread_local int t_handle_release = 0, t_handle_memory = 0;
thread_local bool t_not_idle = false;   // a HandleRelease that could not wait
// Memory freed while waiting was refused (a stream capture in progress, say
// when a garbage collector runs in it): freed by the next HandleRelease that
// could wait.
std::mutex g_late_mu;
std::vector<std::pair<void*, Mem>>& late_frees() {
    static auto* v = new std::vector<std::pair<void*, Mem>>();
    return *v;
}
std::atomic<long long> g_live{0};   // arrays of DevArrays
std::mutex g_heap_mu;
HandleHeap* heaps() {
    static auto* h = new HandleHeap[kMaxDevices];   // outlives every static handle
    return h;
}

cudaMemPool_t pool_of_device() {
    int dev = 0;
    RB_CUDA(cudaGetDevice(&dev));
    RB_REQUIRE(dev >= 0 && dev < kMaxDevices, "device index out of range");
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (!g_pools[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        RB_CUDA(cudaMemPoolCreate(&pool, &props));
        unsigned long long keep = kPoolKeep;
        RB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        g_pools[dev] = pool;
    }
    return g_pools[dev];
}
}  // namespace

bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(s, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone;
}

namespace {
// What the library keeps but does not use goes back to the driver, but for
// some bytes of the pool and of the slabs.
void give_back(size_t keep_pool, size_t keep_slabs) {
    (void)cudaGetLastError();
    RB_CUDA(cudaDeviceSynchronize());
    RB_CUDA(cudaMemPoolTrimTo(pool_of_device(), keep_pool));
    int dev = 0;
    RB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_heap_mu);
    heaps()[dev].trim([](char* base) { cudaFree(base); }, keep_slabs);
}

void* handle_alloc(size_t bytes) {
    int dev = 0;
    RB_CUDA(cudaGetDevice(&dev));
    RB_REQUIRE(dev >= 0 && dev < kMaxDevices, "device index out of range");
    auto get = [](size_t size) {
        void* base = nullptr;
        RB_CUDA(cudaMalloc(&base, size));
        return base;
    };
    {
        std::lock_guard<std::mutex> lock(g_heap_mu);
        try {
            return heaps()[dev].alloc(bytes, get);
        } catch (const Error& e) {
            (void)cudaGetLastError();
            if (e.code != RB_ERR_OOM) throw;
        }
    }
    give_back(0, 0);
    std::lock_guard<std::mutex> lock(g_heap_mu);
    try {
        return heaps()[dev].alloc(bytes, get, 0);   // a slab of this block only
    } catch (...) {
        (void)cudaGetLastError();
        throw;
    }
}
}  // namespace

void trim_memory() { give_back(0, 0); }

void* device_alloc(size_t bytes, Mem* kind) {
    void* p = nullptr;
    cudaStream_t s = stream();
    cudaError_t e;
    if (bytes >= kPoolLargest || capturing(s)) {
        *kind = Mem::kDriver;
        e = cudaMalloc(&p, bytes);
        if (e == cudaErrorMemoryAllocation && !capturing(s)) {   // what is kept may be what is missing
            give_back(0, 0);
            e = cudaMalloc(&p, bytes);
        }
    } else if (t_handle_memory > 0) {
        *kind = Mem::kHandle;
        p = handle_alloc(bytes);
        ++g_live;
        return p;
    } else {
        *kind = Mem::kPool;
        cudaMemPool_t pool = pool_of_device();
        e = cudaMallocFromPoolAsync(&p, bytes, pool, s);
        if (e == cudaErrorMemoryAllocation) {
            give_back(0, 0);
            e = cudaMallocFromPoolAsync(&p, bytes, pool, s);
        }
    }
    if (e != cudaSuccess) (void)cudaGetLastError();
    RB_CUDA(e);
    ++g_live;
    return p;
}

void device_free(void* p, Mem kind) noexcept {
    const bool pooled = kind == Mem::kPool;
    cudaError_t e = cudaErrorUnknown;
    --g_live;
    if (t_handle_release > 0 ? t_not_idle
                             : kind == Mem::kHandle && cudaDeviceSynchronize() != cudaSuccess) {
        (void)cudaGetLastError();
        std::lock_guard<std::mutex> lock(g_late_mu);
        late_frees().emplace_back(p, kind);
        ++g_live;
        return;
    }
    if (kind == Mem::kHandle) {
        std::lock_guard<std::mutex> lock(g_heap_mu);
        for (int d = 0; d < kMaxDevices; d++)
            if (heaps()[d].owns(p)) {
                heaps()[d].free(p, [](char* base) { cudaFree(base); });
                break;
            }
        return;
    }
    if (kind == Mem::kDriver) {
        e = cudaFree(p);
    } else if (t_handle_release > 0) {
        // the device is idle (HandleRelease); a stream the caller set may be
        // gone by now, so the library's own orders the free
        if (g_own_stream || cudaStreamCreateWithFlags(&g_own_stream, cudaStreamNonBlocking) == cudaSuccess)
            e = cudaFreeAsync(p, g_own_stream);
    } else {
        const cudaStream_t s = g_stream ? g_stream : g_own_stream;
        if (s && !capturing(s)) e = cudaFreeAsync(p, s);
    }
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        // (cudaFree does not wait for a pool's memory; where waiting is
        // refused, as in a capture, the memory stays allocated)
        if (pooled && cudaDeviceSynchronize() == cudaSuccess) cudaFree(p);
        (void)cudaGetLastError();
    }
}

HandleRelease::HandleRelease() {
    if (t_handle_release++ > 0) return;
    t_not_idle = cudaDeviceSynchronize() != cudaSuccess;
    if (t_not_idle) {
        (void)cudaGetLastError();
        return;
    }
    std::vector<std::pair<void*, Mem>> late;
    {
        std::lock_guard<std::mutex> lock(g_late_mu);
        late.swap(late_frees());
    }
    for (auto& f : late) device_free(f.first, f.second);
}
HandleRelease::~HandleRelease() {
    if (--t_handle_release > 0) return;
    if (t_not_idle || g_live != 0) return;
    try {
        give_back(kIdleKeep, kIdleSlabs);
    } catch (const std::exception&) {   // no device any more, at process exit
        (void)cudaGetLastError();
    }
}

HandleMemory::HandleMemory() { ++t_handle_memory; }
HandleMemory::~HandleMemory() { --t_handle_memory; }

// Small pinned staging blocks (device scalars read back): cudaMallocHost
// takes over a millisecond, as long as a small setup's kernels, so freed
// blocks are kept for the next handle, at most kPinnedKeep of them.
namespace {
constexpr size_t kPinnedKeep = 16;
std::mutex g_pinned_mu;
std::vector<void*>& pinned_list() {
    static auto* v = new std::vector<void*>();   // outlives every static handle
    return *v;
}
}  // namespace

void* pinned_block() {
    {
        std::lock_guard<std::mutex> lock(g_pinned_mu);
        auto& v = pinned_list();
        if (!v.empty()) {
            void* p = v.back();
            v.pop_back();
            return p;
        }
    }
    void* p = nullptr;
    RB_CUDA(cudaHostAlloc(&p, kPinnedBlock, cudaHostAllocPortable));
    return p;
}

void pinned_release(void* p) noexcept {
    if (!p) return;
    {
        std::lock_guard<std::mutex> lock(g_pinned_mu);
        auto& v = pinned_list();
        if (v.size() < kPinnedKeep) {
            v.push_back(p);
            return;
        }
    }
    cudaFreeHost(p);
}

int sm_count() {
    if (!g_sms) {
        int dev = 0;
        RB_CUDA(cudaGetDevice(&dev));
        RB_CUDA(cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev));
    }
    return g_sms;
}

void tune_cold_l2(const void* warm, size_t bytes) {
    // 192 MB, above the 126 MB L2; allocated once and kept for the process
    constexpr size_t kFlush = (size_t)192 << 20;
    static void* buf = nullptr;
    if (!buf) {
        RB_CUDA(cudaMalloc(&buf, kFlush));
        ++device_alloc_counter();
    }
    RB_CUDA(cudaMemsetAsync(buf, 0, kFlush, stream()));
    if (warm && bytes)
        RB_CUDA(cudaMemcpyAsync(buf, warm, bytes < kFlush ? bytes : kFlush,
                                cudaMemcpyDeviceToDevice, stream()));
}

int resident_blocks_per_sm(const void* fn, int threads) {
    static std::mutex mu;
    static std::unordered_map<const void*, int> cache;
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(fn);
    if (it != cache.end()) return it->second;
    int b = 0;
    RB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, threads, 0));
    if (b < 1) b = 1;
    cache[fn] = b;
    return b;
}

int grid_per_sm(const char* env, int dflt) {
    const char* v = getenv(env);
    const int k = v ? atoi(v) : 0;
    return k > 0 ? k : dflt;
}

rb_csr_s* new_csr(int n_rows, int n_cols, long long nnz) {
    RB_REQUIRE(n_rows >= 0 && n_cols >= 0 && nnz >= 0, "negative matrix dimension");
    RB_REQUIRE(nnz <= INT_MAX, "matrix has more than 2^31-1 nonzeros (int32 indices)");
    auto* A = new rb_csr_s();
    A->n_rows = n_rows;
    A->n_cols = n_cols;
    A->nnz = nnz;
    A->rowptr.alloc((size_t)n_rows + 1);
    A->cols.alloc((size_t)(nnz > 0 ? nnz : 1));
    A->vals.alloc((size_t)(nnz > 0 ? nnz : 1));
    return A;
}

// ------------------------------------------------------------------ scan --
__global__ void k_scan_tail(const int* in, int* out, int n, long long* total) {
    long long t = (n > 0) ? (long long)out[n - 1] + (long long)in[n - 1] : 0;
    *total = t;
    out[n] = (int)t;
}

long long exclusive_scan(const int* in, int* out, int n) {
    if (n == 0) {
        RB_CUDA(cudaMemsetAsync(out, 0, sizeof(int), stream()));
        return 0;
    }
    size_t bytes = 0;
    RB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, n, stream()));
    DevArray<char> tmp(bytes + 16);
    RB_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), bytes, in, out, n, stream()));
    DevArray<long long> tot(1);
    k_scan_tail<<<1, 1, 0, stream()>>>(in, out, n, tot.get());
    RB_CHECK_LAUNCH();
    long long t = read_scalar(tot.get());
    RB_REQUIRE(t >= 0 && t <= INT_MAX, "prefix sum exceeds the int32 index range");
    return t;
}

// -------------------------------------------------- row canonicalisation --
// Each row sorted by column, stably (CSRMatrix::sort, core/matrix.cpp
// :588-618), then the diagonal moved to the front (move_diag_helper,
// :730-786).  G lanes a row read it into shared memory once, and every entry
// finds its place by counting the entries before it, so the row is read and
// written once, coalesced (an insertion sort in global memory, a thread a
// row: 2.97 ms of a 64^3 27-point setup, 0.93 ms its largest call; this way
// 0.29 and 0.13).  Rows longer than the group's share of kSortCap entries are
// then sorted by the whole block, below: an insertion sort by one lane took
// 1.5 s for the column of 9000 entries that a transpose leaves in any order.
constexpr int kSortCap = 384;                    // entries a warp stages (12 bytes each)
constexpr int kSortHalf = 8 * kSortCap / 2;      // a run of a long row: half of what a block stages

// One long row by the block: runs of kSortHalf entries sorted by rank, then
// odd-even rounds that merge neighbouring runs in place (as many rounds as
// runs; pairs in order already are left).  Both are stable, and no scratch
// beyond the block's shared memory is needed.
__device__ void block_sort_row(int i, int s, int m, int* cols, double* vals, int diag_first,
                               double* sv, int* sc) {
    const int tid = threadIdx.x, nth = blockDim.x;
    for (int lo = 0; lo < m; lo += kSortHalf) {
        const int len = min(kSortHalf, m - lo);
        for (int t = tid; t < len; t += nth) {
            sc[t] = cols[s + lo + t];
            sv[t] = vals[s + lo + t];
        }
        __syncthreads();
        for (int t = tid; t < len; t += nth) {
            const int c = sc[t];
            int rank = 0;
            for (int j = 0; j < len; j++) rank += sc[j] < c || (sc[j] == c && j < t);
            cols[s + lo + rank] = c;
            vals[s + lo + rank] = sv[t];
        }
        __syncthreads();
    }
    const int runs = (m + kSortHalf - 1) / kSortHalf;
    for (int round = 0; round < runs; round++)
        for (int r = round & 1; r + 1 < runs; r += 2) {
            const int lo = r * kSortHalf, nr = min(kSortHalf, m - lo - kSortHalf);
            for (int t = tid; t < kSortHalf + nr; t += nth) {
                sc[t] = cols[s + lo + t];
                sv[t] = vals[s + lo + t];
            }
            __syncthreads();
            if (sc[kSortHalf - 1] > sc[kSortHalf])
                for (int t = tid; t < kSortHalf + nr; t += nth) {
                    const int c = sc[t];
                    const bool left = t < kSortHalf;
                    // entries of the other run that come before: smaller
                    // ones, and from the right also equal ones
                    const int* o = left ? sc + kSortHalf : sc;
                    int a = 0, b = left ? nr : kSortHalf;
                    while (a < b) {
                        const int h = (a + b) >> 1;
                        if (o[h] < c || (!left && o[h] == c)) a = h + 1;
                        else b = h;
                    }
                    const int rank = (left ? t : t - kSortHalf) + a;
                    cols[s + lo + rank] = c;
                    vals[s + lo + rank] = sv[t];
                }
            __syncthreads();
        }
    if (!diag_first) return;
    int a = 0, b = m;   // the first entry of the diagonal
    while (a < b) {
        const int h = (a + b) >> 1;
        if (cols[s + h] < i) a = h + 1;
        else b = h;
    }
    const bool has = a < m && cols[s + a] == i;
    const double dv = has ? vals[s + a] : 0.0;
    __syncthreads();
    if (!has) return;
    for (int hi = a; hi > 0; hi -= 2 * kSortHalf) {   // entries before it, one place up
        const int lo = max(0, hi - 2 * kSortHalf);
        for (int t = tid; t < hi - lo; t += nth) {
            sc[t] = cols[s + lo + t];
            sv[t] = vals[s + lo + t];
        }
        __syncthreads();
        for (int t = tid; t < hi - lo; t += nth) {
            cols[s + lo + t + 1] = sc[t];
            vals[s + lo + t + 1] = sv[t];
        }
        __syncthreads();
    }
    if (tid == 0) {
        cols[s] = i;
        vals[s] = dv;
    }
    __syncthreads();
}

template <int G>
__global__ void __launch_bounds__(256)
k_sort_rows(int n, const int* __restrict__ rp, int* cols, double* vals, int diag_first) {
    constexpr int CAP = kSortCap * G / 32;
    __shared__ double sval[8][kSortCap];
    __shared__ int scol[8][kSortCap];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int gl = lane & (G - 1), sub = lane / G;
    const unsigned mask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (lane & ~(G - 1));
    const long i = (((long)blockIdx.x * blockDim.x + threadIdx.x) / G);
    int s = 0, m = 0;
    if (i < n) {
        s = rp[i];
        m = rp[i + 1] - s;
    }
    if (m > 1 && m <= CAP) {
        double* sv = sval[wid] + sub * CAP;
        int* sc = scol[wid] + sub * CAP;
        for (int t = gl; t < m; t += G) {
            sc[t] = cols[s + t];
            sv[t] = vals[s + t];
        }
        __syncwarp(mask);
        for (int t = gl; t < m; t += G) {
            const int c = sc[t];
            int rank = 0, equal_before = 0, diag = 0;
            for (int j = 0; j < m; j++) {
                const int cj = sc[j];
                const int eq = cj == c && j < t;
                rank += cj < c || eq;
                equal_before |= eq;
                diag |= cj == (int)i;
            }
            if (diag_first && diag) {
                if (c == (int)i && !equal_before) rank = 0;
                else if (c < (int)i) rank++;
            }
            cols[s + rank] = c;
            vals[s + rank] = sv[t];
        }
    }
    if (!__syncthreads_or(m > CAP)) return;
    const long first = (long)blockIdx.x * blockDim.x / G;
    for (long k = first; k < first + blockDim.x / G && k < n; k++) {
        const int ks = rp[k], km = rp[k + 1] - ks;
        if (km > CAP) block_sort_row((int)k, ks, km, cols, vals, diag_first, sval[0], scol[0]);
    }
}

void sort_rows_diag_first(rb_csr_s& A, bool diag_first) {
    if (A.n_rows == 0) return;
    // 8 lanes a row up to a mean of 12 entries (prolongators), else 32
    auto go = [&](auto g) {
        constexpr int G = decltype(g)::value;
        k_sort_rows<G><<<grid_for((long)A.n_rows * G, 256), 256, 0, stream()>>>(
            A.n_rows, A.rowptr.get(), A.cols.get(), A.vals.get(), diag_first ? 1 : 0);
    };
    if (A.nnz <= 12LL * A.n_rows) go(std::integral_constant<int, 8>{});
    else go(std::integral_constant<int, 32>{});
    RB_CHECK_LAUNCH();
}

// Deep copy on the device.
rb_csr_s* clone_csr(const rb_csr_s& M) {
    rb_csr_s* C = new_csr(M.n_rows, M.n_cols, M.nnz);
    RB_CUDA(cudaMemcpyAsync(C->rowptr.get(), M.rowptr.get(), sizeof(int) * ((size_t)M.n_rows + 1),
                            cudaMemcpyDeviceToDevice, stream()));
    if (M.nnz) {
        RB_CUDA(cudaMemcpyAsync(C->cols.get(), M.cols.get(), sizeof(int) * M.nnz,
                                cudaMemcpyDeviceToDevice, stream()));
        RB_CUDA(cudaMemcpyAsync(C->vals.get(), M.vals.get(), sizeof(double) * M.nnz,
                                cudaMemcpyDeviceToDevice, stream()));
    }
    return C;
}

// ------------------------------------------------------------ transpose --
__global__ void k_count_cols(long long nnz, const int* __restrict__ cols, int* cnt) {
    long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < nnz) atomicAdd(cnt + cols[j], 1);
}

__global__ void k_scatter_T(int n, const int* __restrict__ rp, const int* __restrict__ cols,
                            const double* __restrict__ vals, int* fill, int* tcols,
                            double* tvals) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int j = rp[i]; j < rp[i + 1]; j++) {
        int c = cols[j];
        int p = atomicAdd(fill + c, 1);
        tcols[p] = i;
        tvals[p] = vals[j];
    }
}

rb_csr_s* transpose(const rb_csr_s& A) {
    rb_csr_s* T = new_csr(A.n_cols, A.n_rows, A.nnz);
    DevArray<int> cnt((size_t)A.n_cols + 1);
    cnt.zero();
    if (A.nnz)
        k_count_cols<<<grid_for(A.nnz, 256), 256, 0, stream()>>>(A.nnz, A.cols.get(), cnt.get());
    RB_CHECK_LAUNCH();
    exclusive_scan(cnt.get(), T->rowptr.get(), A.n_cols);
    RB_CUDA(cudaMemcpyAsync(cnt.get(), T->rowptr.get(), sizeof(int) * A.n_cols,
                            cudaMemcpyDeviceToDevice, stream()));
    if (A.n_rows)
        k_scatter_T<<<grid_for(A.n_rows, 256), 256, 0, stream()>>>(
            A.n_rows, A.rowptr.get(), A.cols.get(), A.vals.get(), cnt.get(), T->cols.get(),
            T->vals.get());
    RB_CHECK_LAUNCH();
    // atomics leave each row in arbitrary order: sort by source row
    sort_rows_diag_first(*T, false);
    return T;
}

// ------------------------------------------------- transposed product --
__global__ void k_iota_vals(long long nnz, double* v) {
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
         k += (long long)gridDim.x * blockDim.x)
        v[k] = (double)k;
}

__global__ void k_to_int(long long nnz, const double* v, int* out) {
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
         k += (long long)gridDim.x * blockDim.x)
        out[k] = (int)v[k];
}

// Rows (or columns, of a transpose map) with more than kLongRow entries: a
// block of their own each, because on a few lanes their load chains outlast
// the whole product (a column of 9000 entries on 8 lanes held a product of
// 5.3M entries at 377 us).  256 entries are 8 batches of 4 on 8 lanes.
constexpr int kLongRow = 256;
constexpr int kRowsLong = 256;   // flag of a handle's lanes value

__global__ void k_long_rows(int n, const int* __restrict__ rp, int* list, int* count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && rp[i + 1] - rp[i] > kLongRow) list[atomicAdd(count, 1)] = i;
}

static void find_long_rows(int n, long long nnz, const int* rp, LongRows& L) {
    L.count = 0;
    if (n == 0 || nnz <= kLongRow) return;
    L.list.alloc((size_t)std::min<long long>(n, nnz / kLongRow));
    DevArray<int> count(1);
    count.zero();
    k_long_rows<<<grid_for(n, 256), 256, 0, stream()>>>(n, rp, L.list.get(), count.get());
    RB_CHECK_LAUNCH();
    L.count = read_scalar(count.get());
    if (!L.count) L.list.release();
}

// Sum of t over a block of kRowBlock threads in a fixed order; thread 0 has it.
__device__ __forceinline__ double block_sum(double t) {
    __shared__ double part[kRowBlock / 32];
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = t;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kRowBlock / 32; w++) s += part[w];
    return s;
}

// The strided row kernel with the long rows on blocks of their own (the
// first nlong of the grid, so that they start at once).
template <int G, class Epi>
__global__ void __launch_bounds__(kRowBlock)
k_csr_rows_long(long n, const int* __restrict__ rp, const int* __restrict__ ci,
                const double* __restrict__ cv, const double* __restrict__ x, Epi epi,
                const int* __restrict__ longs, int nlong) {
    double red = 0.0;
    if ((int)blockIdx.x < nlong) {
        const int row = longs[blockIdx.x];
        const double s = block_sum(row_batched<kRowBlock, RB_ROWS_BATCH, double>(
            rp[row] + (int)threadIdx.x, rp[row + 1], ci, cv, x));
        if (threadIdx.x == 0) epi((long)row, s, red);
        return;
    }
    constexpr int RPW = 32 / G;
    const int lane = threadIdx.x & 31;
    const int sub = lane / G, gl = lane & (G - 1);
    const long gwarp = ((long)(blockIdx.x - nlong) * blockDim.x + threadIdx.x) >> 5;
    const long nwarps = ((long)(gridDim.x - nlong) * blockDim.x) >> 5;
    for (long base = gwarp * RPW; base < n; base += nwarps * RPW) {
        const long row = base + sub;
        int s = 0, e = 0;
        if (row < n) { s = __ldg(rp + row); e = __ldg(rp + row + 1); }
        const bool mine = row < n && e - s <= kLongRow;
        double sum = row_batched<G, RB_ROWS_BATCH, double>(s + gl, mine ? e : s, ci, cv, x);
        sum = group_sum<G>(sum);
        if (mine && gl == 0) epi(row, sum, red);
    }
}

// y_j = sum over the entries of row j of A^T of vals[src] * x[row].  A
// lane's share of a row is walked kTBatch entries at a time: the source
// rows and positions of a batch, then its gathers of vals and x, then the
// products in increasing position, so that the two dependent loads of a
// batch overlap (one entry at a time on 8 lanes, a 27-point row took four
// dependent round trips).  Fixed strides and a fixed shuffle tree: the
// result does not depend on scheduling.
constexpr int kTBatch = 4;
template <int STEP>
__device__ __forceinline__ double t_row(int k, int e, const int* __restrict__ rows,
                                        const int* __restrict__ src,
                                        const double* __restrict__ vals,
                                        const double* __restrict__ x) {
    double s = 0.0;
    for (; k < e; k += kTBatch * STEP) {
        int r[kTBatch], p[kTBatch];
        double v[kTBatch], w[kTBatch];
#pragma unroll
        for (int q = 0; q < kTBatch; q++) {
            const bool ok = k + q * STEP < e;
            r[q] = ok ? __ldg(rows + k + q * STEP) : 0;
            p[q] = ok ? __ldg(src + k + q * STEP) : 0;
        }
#pragma unroll
        for (int q = 0; q < kTBatch; q++) {
            const bool ok = k + q * STEP < e;
            v[q] = ok ? __ldg(vals + p[q]) : 0.0;
            w[q] = ok ? __ldg(x + r[q]) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kTBatch; q++)
            if (k + q * STEP < e) s += v[q] * w[q];
    }
    return s;
}

template <int G>
__global__ void __launch_bounds__(kRowBlock)
k_spmv_T_map(int n, const int* __restrict__ rp, const int* __restrict__ rows,
             const int* __restrict__ src, const double* __restrict__ vals,
             const double* __restrict__ x, double* __restrict__ y, const int* __restrict__ longs,
             int nlong) {
    if ((int)blockIdx.x < nlong) {
        const int j = longs[blockIdx.x];
        const double s = block_sum(t_row<kRowBlock>(rp[j] + (int)threadIdx.x, rp[j + 1], rows, src, vals, x));
        if (threadIdx.x == 0) y[j] = s;
        return;
    }
    const long t = (long)(blockIdx.x - nlong) * blockDim.x + threadIdx.x;
    const long j = t / G;
    const int g = threadIdx.x & (G - 1);
    int b = 0, e = 0;
    if (j < n) { b = __ldg(rp + j); e = __ldg(rp + j + 1); }
    const bool mine = j < n && e - b <= kLongRow;
    double s = t_row<G>(b + g, mine ? e : b, rows, src, vals, x);
    s = group_sum<G>(s);
    if (mine && g == 0) y[j] = s;
}

void spmv_T64(rb_csr_s& A, const double* x, double* y) {
    if (!A.tmap) {
        // transpose a copy of A whose values are the entry positions: the
        // transposed values are then the source positions, in the order the
        // deterministic transpose leaves its rows
        std::unique_ptr<rb_csr_s> I(clone_csr(A));
        if (A.nnz)
            k_iota_vals<<<grid_for(A.nnz, 256), 256, 0, stream()>>>(A.nnz, I->vals.get());
        RB_CHECK_LAUNCH();
        std::unique_ptr<rb_csr_s> T(transpose(*I));
        auto m = std::make_unique<TransposeMap>();
        m->src.alloc((size_t)A.nnz + 1);
        if (A.nnz)
            k_to_int<<<grid_for(A.nnz, 256), 256, 0, stream()>>>(A.nnz, T->vals.get(),
                                                                  m->src.get());
        RB_CHECK_LAUNCH();
        m->rowptr = std::move(T->rowptr);
        m->rows = std::move(T->cols);
        find_long_rows(A.n_cols, A.nnz, m->rowptr.get(), m->longs);
        RB_CUDA(cudaStreamSynchronize(stream()));   // kept on the handle: complete on any stream
        A.tmap = std::move(m);
    }
    if (!A.n_cols) return;
    const TransposeMap& m = *A.tmap;
    auto launch = [&](auto g) {
        constexpr int G = decltype(g)::value;
        k_spmv_T_map<G><<<grid_for((long)A.n_cols * G, kRowBlock) + m.longs.count, kRowBlock, 0, stream()>>>(
            A.n_cols, m.rowptr.get(), m.rows.get(), m.src.get(), A.vals.get(), x, y,
            m.longs.list.get(), m.longs.count);
    };
    // Lanes a row from the mean length.  Measured with 2 / 4 / 8 / 16 lanes
    // (us): 27 entries a row (128^3) 226 / 182 / 199 / 317, 18 (300k ragged
    // rows) 44 / 43 / 46 / 58, 9 (1000^2) 45 / 47 / 73 / 128, 5 within noise;
    // 8 lanes and one entry at a time took 209 us on the first, and 377 us
    // on the second, whose longest row has 9000 entries.
    if ((double)A.nnz > 12.0 * A.n_cols) launch(std::integral_constant<int, 4>{});
    else launch(std::integral_constant<int, 2>{});
    RB_CHECK_LAUNCH();
}

// ---------------------------------------------------------------- dots --
struct FinStore {
    double* out;
    __device__ void operator()(double t) const { *out = t; }
};

__global__ void __launch_bounds__(256) k_dot(const double* __restrict__ a,
                                             const double* __restrict__ b, long n,
                                             ReduceSlot rs, FinStore fin) {
    double t = 0.0;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long)gridDim.x * blockDim.x)
        t += a[i] * b[i];
    block_reduce_finish(t, rs, fin);
}

namespace {
// (memory of the process: never freed, and no array of a handle or a call)
struct ReduceScratch {
    double* partials = nullptr;
    unsigned* ticket = nullptr;
} g_scratch;
}  // namespace

// One scratch for every reduction on the library stream.  It is allocated
// once and never moved, because CUDA graphs capture its address.
constexpr int kMaxReduceGrid = 1 << 16;

ReduceSlot global_reduce_slot(int grid) {
    auto& s = g_scratch;
    RB_REQUIRE(grid <= kMaxReduceGrid, "reduction grid too large");
    if (!s.partials) {
        RB_CUDA(cudaMalloc(&s.ticket, 256 + sizeof(double) * kMaxReduceGrid));
        RB_CUDA(cudaMemsetAsync(s.ticket, 0, sizeof(unsigned), stream()));
        RB_CUDA(cudaStreamSynchronize(stream()));
        s.partials = reinterpret_cast<double*>(reinterpret_cast<char*>(s.ticket) + 256);
        ++device_alloc_counter();
    }
    return ReduceSlot{s.partials, s.ticket};
}

void dot_async(const double* a, const double* b, int n, double* result_dev) {
    const int grid = std::max(1, std::min(sm_count() * 4, (int)((n + 255) / 256)));
    ReduceSlot rs = global_reduce_slot(grid);
    k_dot<<<grid, 256, 0, stream()>>>(a, b, n, rs, FinStore{result_dev});
    RB_CHECK_LAUNCH();
}

// ------------------------------------------------------- FP64 SpMV ops --
void residual64(const CsrView<double>& A, const double* x, const double* b, double* r,
                int lanes) {
    launch_rows(A.rowptr, A.cols, A.vals, A.n_rows, A.nnz, x, EpiResidual<double, double>{b, r},
                lanes);
}

// A handle's products: on the schedule picked for it, with its long rows on
// blocks of their own when that was the fastest (kRowsLong).
template <class Epi>
static void handle_rows(rb_csr_s& A, const double* x, Epi epi, int lanes) {
    if (!(lanes & kRowsLong)) {
        launch_rows(A.rowptr.get(), A.cols.get(), A.vals.get(), A.n_rows, A.nnz, x, epi, lanes);
        return;
    }
    const int nl = A.longs.count;
    auto launch = [&](auto g) {
        constexpr int G = decltype(g)::value;
        k_csr_rows_long<G><<<row_grid(A.n_rows, G) + nl, kRowBlock, 0, stream()>>>(
            A.n_rows, A.rowptr.get(), A.cols.get(), A.vals.get(), x, epi, A.longs.list.get(), nl);
    };
    switch (lanes & (kRowsBlocked - 1)) {
        case 2: launch(std::integral_constant<int, 2>{}); break;
        case 4: launch(std::integral_constant<int, 4>{}); break;
        case 8: launch(std::integral_constant<int, 8>{}); break;
        default: launch(std::integral_constant<int, 16>{}); break;
    }
    RB_CHECK_LAUNCH();
}

void handle_spmv(rb_csr_s& A, const double* x, double* y) {
    handle_rows(A, x, EpiStore<double>{y}, handle_lanes(A, x));
}
void handle_residual(rb_csr_s& A, const double* x, const double* b, double* r) {
    handle_rows(A, x, EpiResidual<double, double>{b, r}, handle_lanes(A, x));
}
void handle_append(rb_csr_s& A, const double* x, double* y) {
    handle_rows(A, x, EpiAppend<double>{y}, handle_lanes(A, x));
}

int handle_lanes(rb_csr_s& A, const double* x) {
    if (A.lanes) return A.lanes;
    if (A.n_rows < 4096 || A.nnz == 0) return A.lanes = pick_group(A.n_rows, A.nnz);
    // products into a scratch vector of its own (the caller's output may be
    // an input too, as in mult_append), each schedule timed over 3 launches
    DevArray<double> y((size_t)A.n_rows);
    static const int cands[10] = {2, 4, 8, 16, 32, kRowsBlocked | 4, kRowsBlocked | 8,
                                  kRowsBlocked | 16, kRowsBlocked | 32, 1};
    cudaEvent_t e0, e1;
    RB_CUDA(cudaEventCreate(&e0));
    RB_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    int bestG = pick_group(A.n_rows, A.nnz);
    std::vector<int> tries(cands, cands + 10);
    find_long_rows(A.n_rows, A.nnz, A.rowptr.get(), A.longs);
    if (A.longs.count)
        for (int G : {2, 4, 8, 16}) tries.push_back(kRowsLong | G);
    const EpiStore<double> out{y.get()};
    for (int G : tries) {
        handle_rows(A, x, out, G);
        RB_CUDA(cudaEventRecord(e0, stream()));
        for (int rep = 0; rep < 3; rep++) handle_rows(A, x, out, G);
        RB_CUDA(cudaEventRecord(e1, stream()));
        RB_CUDA(cudaEventSynchronize(e1));
        float ms = 0;
        RB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (ms < best) { best = ms; bestG = G; }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return A.lanes = bestG;
}

}  // namespace rb
