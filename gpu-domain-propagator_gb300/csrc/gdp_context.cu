// gdp_context.cu -- host side of the propagator: input validation, device
// layout (SELL slices of thread rows, warp tiles of split rows, work items,
// marking index), device buffers and the three round-loop drivers.
//
// Replaces the reference's per-call host driver propagateConstraintsGPUAtomic
// (src/propagators/GPU_propagator.cuh:98-268): uploads, row binning
// (fill_row_blocks, src/kernels/util_kernels.cu:12-62) and the round loops
// (CPU_LOOP :160-204, GPU_LOOP :146-159, MEGAKERNEL :205-255). CUDA errors
// return GDP_ERROR with a message instead of exit() (src/cuda_def.cuh:10-15).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <thread>
#include <vector>
#ifdef GDP_BUILD_TIMERS
#include <chrono>
#include <cstdio>
#endif

#ifdef _OPENMP
#include <omp.h>
#endif

#include "gdp_context.h"
#include "gdp_device.cuh"
#include "gdp_learned.h"
#include "gdp_sequence.h"

namespace gdp {

namespace {
thread_local std::string g_last_error;

// Allocator that leaves the elements of a resized vector uninitialised: the
// layout's per-row host arrays are written in full by parallel loops, and
// zero-filling them first cost a serial pass over megabytes.
template <class T>
struct NoInit : std::allocator<T> {
    template <class U>
    struct rebind {
        using other = NoInit<U>;
    };
    NoInit() = default;
    template <class U>
    NoInit(const NoInit<U> &) {}
    template <class U>
    void construct(U *p) {
        ::new ((void *)p) U;
    }
    template <class U, class... A>
    void construct(U *p, A &&...a) {
        ::new ((void *)p) U(std::forward<A>(a)...);
    }
};
template <class T>
using RawVec = std::vector<T, NoInit<T>>;

// Build stamps, compiled only into a library built with -DGDP_BUILD_TIMERS
// (build.py --build-timers): host wall-clock times of Context::init's
// milestones (ms since it began) and device times of the raw CSR upload and
// the layout kernels, printed to stderr when a build ends. In the plain build
// every call is empty.
struct BuildStamps {
#ifdef GDP_BUILD_TIMERS
    std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
    double host[7] = {};
    cudaEvent_t ev[4] = {};  // upload begins / ends (helper stream), layout begins / ends
    void mark(int k) {
        host[k] = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
    void record(int k, cudaStream_t s) {
        if (!ev[k]) cudaEventCreate(&ev[k]);
        cudaEventRecord(ev[k], s);
    }
    void report() {
        float up = 0.f, start = 0.f, lay = 0.f;
        if (ev[0] && ev[1]) cudaEventElapsedTime(&up, ev[0], ev[1]);
        if (ev[0] && ev[2]) cudaEventElapsedTime(&start, ev[0], ev[2]);
        if (ev[2] && ev[3]) cudaEventElapsedTime(&lay, ev[2], ev[3]);
        fprintf(stderr,
                "gdp build (ms): validated %.2f set-up %.2f binned %.2f joined %.2f launched %.2f queued %.2f "
                "synced %.2f | device: upload %.2f, layout starts %.2f after the upload began, layout %.2f\n",
                host[0], host[1], host[2], host[3], host[4], host[5], host[6], up, start, lay);
    }
    ~BuildStamps() {
        for (cudaEvent_t e : ev)
            if (e) cudaEventDestroy(e);
    }
#else
    void mark(int) {}
    void record(int, cudaStream_t) {}
    void report() {}
#endif
};
}

void set_error(const std::string &msg) { g_last_error = msg; }
const char *last_error() { return g_last_error.c_str(); }

#define GDP_CUDA(expr)                                                                  \
    do {                                                                                \
        cudaError_t e_ = (cudaError_t)(expr);                                           \
        if (e_ != cudaSuccess) {                                                        \
            set_error(std::string(#expr) + " failed: " + cudaGetErrorString(e_));       \
            return GDP_ERROR;                                                           \
        }                                                                               \
    } while (0)

// ---------------------------------------------------------------------------
namespace {
// Device blocks of released arenas by (device, size). A request takes the
// smallest cached block of its device that is at least as large and at most
// 5/4 of the request. The cache keeps at most kCacheMax bytes; blocks beyond
// that are freed. The object is never destroyed: at exit the CUDA runtime
// may be gone before static destructors run, and the driver reclaims the
// memory anyway.
struct BlockCache {
    std::mutex mu;
    std::multimap<std::pair<int, size_t>, void *> blocks;
    size_t bytes = 0;
};
constexpr size_t kCacheMax = size_t(32) << 30;
BlockCache &block_cache() {
    static BlockCache *c = new BlockCache;
    return *c;
}
}  // namespace

void release_cached_memory() {
    BlockCache &c = block_cache();
    std::lock_guard<std::mutex> g(c.mu);
    int cur = 0;
    cudaGetDevice(&cur);
    for (const auto &kv : c.blocks) {
        cudaSetDevice(kv.first.first);
        cudaFree(kv.second);
    }
    cudaSetDevice(cur);
    cudaGetLastError();
    c.blocks.clear();
    c.bytes = 0;
}


// Streams, events and page-locked memory of destroyed contexts, kept for later
// ones: creating and destroying them takes about 250 us, half the time of a
// context of 100 rows. At most kKeptResources sets are kept (any thread takes
// and gives them back); the object is never destroyed, as above.
namespace {
constexpr size_t kKeptResources = 16;
struct ResourcePool {
    std::mutex mu;
    std::vector<HostResources *> free;
};
ResourcePool &resource_pool() {
    static ResourcePool *p = new ResourcePool;
    return *p;
}
void destroy_resources(HostResources *r) {
    if (r->ev0) cudaEventDestroy(r->ev0);
    if (r->ev1) cudaEventDestroy(r->ev1);
    if (r->uploaded) cudaEventDestroy(r->uploaded);
    if (r->pinned) cudaFreeHost(r->pinned);
    if (r->stream) cudaStreamDestroy(r->stream);
    if (r->upload) cudaStreamDestroy(r->upload);
    delete r;
}
}  // namespace

// The caller has set the device; null (and the error) on failure.
HostResources *take_resources(int device, cudaError_t *err) {
    ResourcePool &pool = resource_pool();
    {
        std::lock_guard<std::mutex> g(pool.mu);
        for (size_t i = pool.free.size(); i-- > 0;)
            if (pool.free[i]->device == device) {
                HostResources *r = pool.free[i];
                pool.free.erase(pool.free.begin() + (long)i);
                return r;
            }
    }
    HostResources *r = new HostResources;
    r->device = device;
    cudaError_t e = cudaStreamCreateWithFlags(&r->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&r->upload, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&r->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&r->ev1);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&r->uploaded, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaMallocHost(&r->pinned, HostResources::kFlagBytes + HostResources::kStageBytes);
    if (e != cudaSuccess) {
        destroy_resources(r);
        *err = e;
        return nullptr;
    }
    return r;
}

// Both streams are waited for: a later owner finds them empty.
void give_resources(HostResources *r) {
    if (!r) return;
    const bool idle = cudaStreamSynchronize(r->stream) == cudaSuccess && cudaStreamSynchronize(r->upload) == cudaSuccess;
    cudaGetLastError();
    ResourcePool &pool = resource_pool();
    {
        std::lock_guard<std::mutex> g(pool.mu);
        if (idle && pool.free.size() < kKeptResources) {
            pool.free.push_back(r);
            return;
        }
    }
    destroy_resources(r);
}

void release_kept_resources() {
    ResourcePool &pool = resource_pool();
    std::vector<HostResources *> free;
    {
        std::lock_guard<std::mutex> g(pool.mu);
        free.swap(pool.free);
    }
    for (HostResources *r : free) destroy_resources(r);
    cudaGetLastError();
}

Arena::~Arena() { release(); }

void Arena::release() {
    if (blocks.empty()) return;
    // a block may still be read by work on any stream of its device (the
    // device-pointer entry points take the caller's stream): wait for the
    // device, as cudaFree would
    int cur = 0;
    cudaGetDevice(&cur);
    int synced = -1;
    for (const Block &b : blocks)
        if (b.dev != synced) {
            cudaSetDevice(b.dev);
            cudaDeviceSynchronize();
            synced = b.dev;
        }
    cudaSetDevice(cur);
    cudaGetLastError();
    BlockCache &c = block_cache();
    std::lock_guard<std::mutex> g(c.mu);
    for (const Block &b : blocks) {
        if (c.bytes + b.bytes <= kCacheMax) {
            c.blocks.emplace(std::make_pair(b.dev, b.bytes), b.p);
            c.bytes += b.bytes;
        } else {
            cudaFree(b.p);
        }
    }
    blocks.clear();
}

void *Arena::alloc_bytes(size_t bytes) {
    bytes = (std::max<size_t>(bytes, 1) + 255) & ~size_t(255);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    {
        BlockCache &c = block_cache();
        std::lock_guard<std::mutex> g(c.mu);
        auto it = c.blocks.lower_bound(std::make_pair(dev, bytes));
        if (it != c.blocks.end() && it->first.first == dev && it->first.second - bytes <= bytes / 4) {
            const Block blk{it->second, it->first.second, dev};
            c.blocks.erase(it);
            c.bytes -= blk.bytes;
            blocks.push_back(blk);
            return blk.p;
        }
    }
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {  // the cache may hold the memory: free it, retry once
        cudaGetLastError();
        release_cached_memory();
        if (cudaMalloc(&p, bytes) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
    }
    blocks.push_back(Block{p, bytes, dev});
    return p;
}

bool Arena::carve(std::initializer_list<Piece> pieces) {
    size_t total = 0;
    for (const Piece &p : pieces) total += (std::max<size_t>(p.bytes, 1) + 255) & ~size_t(255);
    unsigned char *d = (unsigned char *)alloc_bytes(total);
    if (!d) return false;
    for (const Piece &p : pieces) {
        *p.dst = d;
        d += (std::max<size_t>(p.bytes, 1) + 255) & ~size_t(255);
    }
    return true;
}

namespace {
// Host arrays gathered and sent by send(): one device block and, with room in a
// page-locked stage, one copy.
struct Uploads {
    struct Part {
        const void *src;
        size_t bytes, at;
        void **dst;
    };
    std::vector<Part> parts;
    size_t total = 0;
    template <class T>
    void add(T *&dst, const void *src, size_t bytes) {
        parts.push_back(Part{src, bytes, total, (void **)&dst});
        total += (std::max<size_t>(bytes, 1) + 255) & ~size_t(255);
    }
    // false: no memory, or a copy failed
    bool send(Arena &arena, cudaStream_t s, unsigned char *stage, size_t stage_bytes) {
        unsigned char *d = (unsigned char *)arena.alloc_bytes(total);
        if (!d) return false;
        const bool packed = stage && total <= stage_bytes;
        for (const Part &p : parts) {
            *p.dst = d + p.at;
            if (!p.bytes) continue;
            if (packed) std::memcpy(stage + p.at, p.src, p.bytes);
            else if (cudaMemcpyAsync(d + p.at, p.src, p.bytes, cudaMemcpyHostToDevice, s) != cudaSuccess) return false;
        }
        if (packed && cudaMemcpyAsync(d, stage, total, cudaMemcpyHostToDevice, s) != cudaSuccess) return false;
        parts.clear();
        total = 0;
        return true;
    }
};
}  // namespace

// ---------------------------------------------------------------------------
// The checks that make the raw arrays safe to copy: sizes, pointers and the
// row pointer's end points.
static GDP_RETCODE validate_shape(int m, int n, int nnz, const int *col, const int *row_ptr, const double *val,
                                  const int *vartype) {
    if (m < 0 || n < 0 || nnz < 0) { set_error("negative problem size"); return GDP_ERROR; }
    if (!col || !row_ptr || !val || !vartype) { set_error("null input array"); return GDP_ERROR; }
    if (row_ptr[0] != 0 || row_ptr[m] != nnz) {
        set_error("csr_row_ptrs must start at 0 and end at nnz");
        return GDP_ERROR;
    }
    return GDP_OKAY;
}

// Host threads for a loop over `items` rows or variables: one per 32K, so a
// small problem starts none (waking 15 threads takes 10 to 50 us a loop, and
// milliseconds when one of them is descheduled); one core is left to the
// upload's helper thread.
static int host_threads_for(long long items) {
#ifdef _OPENMP
    return (int)std::max(1LL, std::min<long long>(items >> 15, omp_get_max_threads() - 1));
#else
    return 1;
#endif
}

GDP_RETCODE validate_csr(int m, int n, int nnz, const int *col, const int *row_ptr,
                         const double *val, const int *vartype) {
    if (validate_shape(m, n, nnz, col, row_ptr, val, vartype) != GDP_OKAY) return GDP_ERROR;
    int bad_row = INT_MAX, bad_var = INT_MAX;
#pragma omp parallel for reduction(min : bad_row) schedule(static) num_threads(host_threads_for(m))
    for (int i = 0; i < m; i++)
        if (row_ptr[i + 1] < row_ptr[i]) bad_row = std::min(bad_row, i);
    if (bad_row != INT_MAX) { set_error("csr_row_ptrs is not monotone"); return GDP_ERROR; }
#pragma omp parallel for reduction(min : bad_var) schedule(static) num_threads(host_threads_for(n))
    for (int j = 0; j < n; j++)
        if (vartype[j] != 0 && vartype[j] != 1 && vartype[j] != 3) bad_var = std::min(bad_var, j);
    if (bad_var != INT_MAX) {
        set_error("vartype must be 0, 1 or 3 (variable " + std::to_string(bad_var) + ")");
        return GDP_ERROR;
    }
    return GDP_OKAY;
}

// The element checks (column range, finite coefficients) run on the device
// over the uploaded raw CSR; this turns their result into the error.
static GDP_RETCODE element_error(const int bad[2]) {
    if (bad[0] != INT_MAX) {
        set_error("column index out of range at non-zero " + std::to_string(bad[0]));
        return GDP_ERROR;
    }
    if (bad[1] != INT_MAX) {
        set_error("non-finite coefficient at non-zero " + std::to_string(bad[1]));
        return GDP_ERROR;
    }
    return GDP_OKAY;
}

// ---------------------------------------------------------------------------
GDP_RETCODE Context::init(int m_, int n_, int nnz_, const int *col, const int *row_ptr,
                          const double *val, const double *lhs, const double *rhs,
                          const int *vartype, const gdp_options *o) {
    m = m_; n = n_; nnz = nnz_;
    gdp_default_options(&opts);
    if (o) opts = *o;
    if (opts.max_rounds <= 0) opts.max_rounds = GDP_MAX_NUM_ROUNDS;
    if (opts.thread_row_max <= 0) opts.thread_row_max = 32;
    if (opts.split_tile <= 0) opts.split_tile = 1024;
    if (opts.use_marking < 0) opts.use_marking = 1;
    if (opts.thread_row_max > (1 << 20)) opts.thread_row_max = 1 << 20;
    if (opts.split_tile > (1 << 24)) opts.split_tile = 1 << 24;
    if (opts.sync_type < CPU_LOOP || opts.sync_type > MEGAKERNEL) {
        set_error("Unknown sync type");
        return GDP_ERROR;
    }
    if (opts.cta_threads != 0 && opts.cta_threads != 128 && opts.cta_threads != 256 && opts.cta_threads != 512) {
        set_error("cta_threads must be 128, 256 or 512");
        return GDP_ERROR;
    }
    if (!lhs || !rhs) { set_error("null lhs/rhs"); return GDP_ERROR; }
    BuildStamps stamps;
    if (validate_csr(m, n, nnz, col, row_ptr, val, vartype) != GDP_OKAY) return GDP_ERROR;  // host part
    stamps.mark(0);

    GDP_CUDA(cudaSetDevice(opts.device));
    cudaGetLastError();  // every call below is checked; start from a clean error state
    {
        cudaError_t e = cudaSuccess;
        res = take_resources(opts.device, &e);
        if (!res) GDP_CUDA(e);
    }
    stream = res->stream;
    ev0 = res->ev0;
    ev1 = res->ev1;
    h_flags = reinterpret_cast<RoundFlags *>(res->pinned);
    int sms = 0;
    GDP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, opts.device));
    n_sms = sms;
    int pageable = 0;
    GDP_CUDA(cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, opts.device));
    host_direct = pageable == 1;

    // The raw CSR goes up from a helper thread, on a stream of its own, while
    // this thread bins the rows: a copy from pageable memory returns only
    // once its source has been staged, so issuing it here would serialise
    // the two. This thread makes no CUDA call until the row layout is
    // decided (the driver would hold it while the copy runs). The helper
    // leaves once the copies are queued; the layout build that reads them
    // waits for them on the device (an event), after the join. The element
    // checks (column range, finite coefficients) run on the device over the
    // copies.
    // A small problem takes no helper: its arrays and the layout's are packed
    // into the page-locked stage and go up in one copy.
    stamps.mark(1);
    const size_t raw_bytes = sizeof(int) * (size_t)nnz + sizeof(double) * (size_t)nnz + sizeof(int) * ((size_t)m + 1) +
                             2 * sizeof(double) * (size_t)m;
    // the layout's arrays are at most about 100 bytes per row and tile, and a byte per variable
    const bool small = raw_bytes + 128 * (size_t)m + 2 * (size_t)n + 16384 <= HostResources::kStageBytes;
    Arena raw;  // raw CSR and row sides, released when the build is done
    int *dcol = nullptr, *drp = nullptr;
    double *dval = nullptr, *dlhs = nullptr, *drhs = nullptr;
    std::string up_err;
    struct UploadStream {  // the helper's stream
        cudaStream_t s = nullptr;
        ~UploadStream() {
            if (s) cudaStreamSynchronize(s);  // before the raw buffers can be freed
        }
    } ups;
    // marking index (variable -> row positions, |a| rounded up): the helper
    // counts the columns as soon as they are up; the layout kernels fill it
    const size_t n1 = (size_t)n + 1;
    int *vp = (int *)arena.alloc_bytes(sizeof(int) * n1);
    VarEntry *vent = (VarEntry *)arena.alloc_bytes(sizeof(VarEntry) * (size_t)std::max(nnz, 1));
    int *vcur = (int *)raw.alloc_bytes(sizeof(int) * n1);
    int *vscan = (int *)raw.alloc_bytes(sizeof(int) * ((n1 + 1023) / 1024 + 1));
    if (!vp || !vent || !vcur || !vscan) {
        set_error("device allocation failed (marking index)");
        return GDP_ERROR;
    }
    struct Joined {
        std::thread t;
        ~Joined() {
            if (t.joinable()) t.join();
        }
    } uploader;  // declared after everything the thread touches: joined first
    if (!small) {
        ups.s = res->upload;
        uploader.t = std::thread([&, dev = opts.device] {
            auto fail = [&](const char *what, cudaError_t e) {
                up_err = std::string(what) + ": " + cudaGetErrorString(e);
                cudaGetLastError();
            };
            cudaError_t e = cudaSetDevice(dev);
            if (e != cudaSuccess) return fail("cudaSetDevice", e);
            const size_t nz = (size_t)std::max(nnz, 1);
            dcol = (int *)raw.alloc_bytes(sizeof(int) * nz);
            dval = (double *)raw.alloc_bytes(sizeof(double) * nz);
            drp = (int *)raw.alloc_bytes(sizeof(int) * ((size_t)m + 1));
            dlhs = (double *)raw.alloc_bytes(sizeof(double) * (size_t)std::max(m, 1));
            drhs = (double *)raw.alloc_bytes(sizeof(double) * (size_t)std::max(m, 1));
            if (!dcol || !dval || !drp || !dlhs || !drhs) {
                up_err = "device allocation failed (raw CSR)";
                return;
            }
            cudaStream_t us = ups.s;
            stamps.record(0, us);
            if (nnz) e = cudaMemcpyAsync(dcol, col, sizeof(int) * (size_t)nnz, cudaMemcpyHostToDevice, us);
            if (e == cudaSuccess && nnz)
                e = cudaMemcpyAsync(dval, val, sizeof(double) * (size_t)nnz, cudaMemcpyHostToDevice, us);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(drp, row_ptr, sizeof(int) * ((size_t)m + 1), cudaMemcpyHostToDevice, us);
            if (e == cudaSuccess && m) e = cudaMemcpyAsync(dlhs, lhs, sizeof(double) * (size_t)m, cudaMemcpyHostToDevice, us);
            if (e == cudaSuccess && m) e = cudaMemcpyAsync(drhs, rhs, sizeof(double) * (size_t)m, cudaMemcpyHostToDevice, us);
            stamps.record(1, us);
            if (e == cudaSuccess) e = (cudaError_t)build_marking_counts(dcol, nnz, n, vp, vcur, vscan, us);
            if (e == cudaSuccess) e = cudaEventRecord(res->uploaded, us);
            if (e != cudaSuccess) fail("raw CSR upload", e);
        });
    }

    const int host_threads = host_threads_for(m);
    // ---- row binning (SELL-g) ----
    // g = 1 for rows up to thread_row_max; g = smallest power of two >= len/32
    // (2..32) up to split_tile; longer rows are split into warp tiles.
    const int Lt = opts.thread_row_max, Ls = std::max(opts.split_tile, Lt);
    auto lanes_of = [&](int L) {
        if (L <= Lt) return 1;
        int g = 2;
        while (g < 32 && g * 32 < L) g <<= 1;
        return g;
    };
    std::unique_ptr<int[]> len(new int[std::max(m, 1)]);
    int lmax = 0;  // longest SELL row
#pragma omp parallel for reduction(max : lmax) schedule(static) num_threads(host_threads)
    for (int i = 0; i < m; i++) {
        len[i] = row_ptr[i + 1] - row_ptr[i];
        if (len[i] <= Ls) lmax = std::max(lmax, len[i]);
    }
    // SELL rows (1..Ls non-zeros) by lanes per row (widest first), then length
    // (longest first), stable: lanes_of never decreases with the length, so
    // this is a counting sort by length, longest first -- run in parallel over
    // contiguous row chunks (per-chunk histograms keep it stable; a team may have
    // fewer threads than there are chunks). Split rows
    // (longer than Ls) are collected in row order and sorted by length.
    // pos_row: the original row of every position -- SELL positions first (the
    // row order the layout is built from), then the split rows; uploaded as is
    RawVec<int> pos_row((size_t)std::max(m, 1));
    std::vector<int> split_rows;
    // per SELL row length L: first position, and first element of the
    // row-contiguous copy (rows of one length are consecutive positions)
    std::vector<int> len_start((size_t)lmax + 1, 0);
    std::vector<long long> len_base((size_t)lmax + 1, 0);
    long long x_elems = 0;  // elements of the row-contiguous copy
    int n_sell_rows = 0;
    {
#ifdef _OPENMP
        const int nt = lmax <= (1 << 16) ? std::min(host_threads, 64) : 1;
#else
        const int nt = 1;
#endif
        const size_t W = (size_t)lmax + 1;  // keys 0..lmax (0: empty rows, skipped)
        std::vector<int> hist((size_t)nt * W, 0);
        std::vector<int> nsplit(nt + 1, 0);
#pragma omp parallel for schedule(static, 1) num_threads(nt)
        for (int t = 0; t < nt; t++) {
            const int i0 = (int)((long long)m * t / nt), i1 = (int)((long long)m * (t + 1) / nt);
            int *h = &hist[(size_t)t * W];
            for (int i = i0; i < i1; i++) {
                if (len[i] > Ls) nsplit[t + 1]++;
                else h[len[i]]++;
            }
        }
        // offsets: longer rows first; within a length, chunks in row order
        int acc = 0;
        for (int L = lmax; L >= 1; L--) {
            len_start[L] = acc;
            len_base[L] = x_elems;
            for (int t = 0; t < nt; t++) {
                const int c = hist[(size_t)t * W + L];
                hist[(size_t)t * W + L] = acc;
                acc += c;
            }
            x_elems += (long long)(acc - len_start[L]) * ((L + 3) & ~3);  // rows start on 4-element boundaries
        }
        for (int t = 0; t < nt; t++) nsplit[t + 1] += nsplit[t];
        n_sell_rows = acc;
        split_rows.resize(nsplit[nt]);
#pragma omp parallel for schedule(static, 1) num_threads(nt)
        for (int t = 0; t < nt; t++) {
            const int i0 = (int)((long long)m * t / nt), i1 = (int)((long long)m * (t + 1) / nt);
            int *h = &hist[(size_t)t * W];
            int sp = nsplit[t];
            for (int i = i0; i < i1; i++) {
                if (len[i] > Ls) split_rows[sp++] = i;
                else if (len[i] > 0) pos_row[h[len[i]]++] = i;
            }
        }
    }
    std::stable_sort(split_rows.begin(), split_rows.end(), [&](int a, int b) { return len[a] > len[b]; });
    const int ns = n_sell_rows;
    const int *order = pos_row.data();  // row position -> original row

    n_srows = ns;
    // slices: the rows of one lanes-per-row class are consecutive positions;
    // a class of g lanes is cut into slices of 32 / g rows, each as wide as
    // its first (longest) row
    std::vector<long long> slice_ptr;
    std::vector<int> slice_row0, slice_lg;
    int g1_begin = ns;  // first position of the one-lane rows
    {
        int cls_lo[6], cls_hi[6], cls_first[6];
        for (int c = 0; c < 6; c++) { cls_lo[c] = 0; cls_hi[c] = 0; }
        for (int p = 0; p < ns;) {  // class boundaries: binary search on the sorted lengths
            const int g = lanes_of(len[order[p]]);
            int lg = 0;
            while ((1 << lg) < g) lg++;
            int lo = p, hi = ns;  // first position of a smaller class
            while (lo < hi) {
                const int mid = lo + (hi - lo) / 2;
                if (lanes_of(len[order[mid]]) == g) lo = mid + 1;
                else hi = mid;
            }
            cls_lo[lg] = p;
            cls_hi[lg] = lo;
            p = lo;
        }
        if (cls_hi[0] > cls_lo[0]) g1_begin = cls_lo[0];
        int nsl = 0;
        for (int lg = 5; lg >= 0; lg--) {
            cls_first[lg] = nsl;
            const int per = 32 >> lg;
            nsl += (cls_hi[lg] - cls_lo[lg] + per - 1) / per;
        }
        slice_row0.resize((size_t)nsl + 1);
        slice_lg.resize((size_t)std::max(nsl, 1), 0);
        slice_ptr.resize((size_t)nsl + 1);
        std::vector<long long> width((size_t)std::max(nsl, 1), 0);
        for (int lg = 5; lg >= 0; lg--) {
            const int per = 32 >> lg, g = 1 << lg, c0 = cls_lo[lg], c1 = cls_hi[lg];
            const int k_n = (c1 - c0 + per - 1) / per;
#pragma omp parallel for schedule(static) num_threads(host_threads)
            for (int k = 0; k < k_n; k++) {
                const int s = cls_first[lg] + k, r0 = c0 + k * per;
                slice_row0[s] = r0;
                slice_lg[s] = lg;
                width[s] = (len[order[r0]] + g - 1) / g;
            }
        }
        slice_row0[nsl] = ns;
        slice_ptr[0] = 0;
        for (int s = 0; s < nsl; s++) slice_ptr[s + 1] = slice_ptr[s] + 32LL * width[s];
        n_slices = nsl;
    }
    sell_elems = slice_ptr[n_slices];
    // per row position (length, sides, first element of the row-contiguous
    // copy, slice): built on the device from the row order
    // split rows: CSR-contiguous, warp tiles of split_tile non-zeros
    n_lrows = (int)split_rows.size();
    std::vector<long long> lrow_ptr(n_lrows + 1, 0);
    std::vector<int> lrow_tile0(n_lrows + 1, 0);
    std::vector<double> lrow_lhs(std::max(n_lrows, 1)), lrow_rhs(std::max(n_lrows, 1));
    std::vector<int> tile_row, tile_begin, tile_end;
    {  // element and tile offsets (prefix sums), then the row sides and tiles in parallel
        const long long tl = opts.split_tile;
        for (int r = 0; r < n_lrows; r++) {
            const int L = len[split_rows[r]];
            lrow_ptr[r + 1] = lrow_ptr[r] + L;
            lrow_tile0[r + 1] = lrow_tile0[r] + (int)((L + tl - 1) / tl);
        }
        n_tiles = lrow_tile0[n_lrows];
        tile_row.resize(n_tiles);
        tile_begin.resize(n_tiles);
        tile_end.resize(n_tiles);
#pragma omp parallel for schedule(static) num_threads(host_threads)
        for (int r = 0; r < n_lrows; r++) {
            const int i = split_rows[r];
            lrow_lhs[r] = lhs[i];
            lrow_rhs[r] = rhs[i];
            int t = lrow_tile0[r];
            for (long long b = lrow_ptr[r]; b < lrow_ptr[r + 1]; b += tl, t++) {
                tile_row[t] = r;
                tile_begin[t] = (int)b;
                tile_end[t] = (int)std::min(b + tl, lrow_ptr[r + 1]);
            }
        }
    }
    const long long lnnz = lrow_ptr[n_lrows];
    // work items of the activity phase, heaviest first (slices: 32 x width non-zeros)
    std::vector<int> items;
    items.reserve((size_t)n_slices + n_tiles);
    {
        std::vector<std::pair<long long, int>> cost;
        cost.reserve((size_t)n_slices + n_tiles);
        long long wmax = 0;
        for (int s = 0; s < n_slices; s++) cost.emplace_back(slice_ptr[s + 1] - slice_ptr[s], s);
        for (int t = 0; t < n_tiles; t++) cost.emplace_back((long long)(tile_end[t] - tile_begin[t]), -t - 1);
        for (auto &c : cost) wmax = std::max(wmax, c.first);
        if (wmax <= (1 << 20)) {  // stable counting sort, heaviest first
            std::vector<int> start((size_t)wmax + 2, 0);
            for (auto &c : cost) start[c.first]++;
            int acc = 0;
            for (long long w = wmax; w >= 0; w--) {
                const int k = start[w];
                start[w] = acc;
                acc += k;
            }
            items.resize(cost.size());
            for (auto &c : cost) items[start[c.first]++] = c.second;
        } else {
            std::stable_sort(cost.begin(), cost.end(),
                             [](const std::pair<long long, int> &a, const std::pair<long long, int> &b) {
                                 return a.first > b.first;
                             });
            for (auto &c : cost) items.push_back(c.second);
        }
    }
    // ---- upload ----
    Uploads ups1, ups2;  // what the layout build reads; the rest
    unsigned char *stage = small ? (unsigned char *)res->pinned + HostResources::kFlagBytes : nullptr;
#define GDP_UP(dst, vec) ups1.add(dst, (vec).data(), sizeof((vec)[0]) * (vec).size())
    std::memset(&P, 0, sizeof(P));
    P.n = n;
    P.n_srows = n_srows;
    P.n_slices = n_slices;
    GDP_UP(P.slice_ptr, slice_ptr);
    GDP_UP(P.slice_row0, slice_row0);
    GDP_UP(P.slice_lg, slice_lg);
    stamps.mark(2);
    int *d_srow_len, *d_xptr, *d_pos_slice;
    double *d_srow_lhs, *d_srow_rhs;
    if (!arena.carve({{(void **)&d_srow_len, sizeof(int) * (size_t)ns},
                      {(void **)&d_xptr, sizeof(int) * (size_t)ns},
                      {(void **)&d_pos_slice, sizeof(int) * (size_t)ns},
                      {(void **)&d_srow_lhs, sizeof(double) * (size_t)ns},
                      {(void **)&d_srow_rhs, sizeof(double) * (size_t)ns}})) {
        set_error("device allocation failed (row positions)");
        return GDP_ERROR;
    }
    P.srow_len = d_srow_len;
    P.xptr = d_xptr;
    P.pos_slice = d_pos_slice;
    P.srow_lhs = d_srow_lhs;
    P.srow_rhs = d_srow_rhs;
    P.n_lrows = n_lrows;
    P.n_tiles = n_tiles;
    GDP_UP(P.lrow_lhs, lrow_lhs);
    GDP_UP(P.lrow_rhs, lrow_rhs);
    GDP_UP(P.lrow_tile0, lrow_tile0);
    if (tile_row.empty()) { tile_row.push_back(0); tile_begin.push_back(0); tile_end.push_back(0); }
    GDP_UP(P.tile_row, tile_row);
    GDP_UP(P.tile_begin, tile_begin);
    GDP_UP(P.tile_end, tile_end);
    // The device builds the layout and then the marking index while this
    // thread prepares the rest (row origins, work lists, variable types) and
    // sends it up on the helper's stream; one synchronisation at the end, then
    // the element checks' verdict.
    Arena tmp;  // the row maps, freed when the build is done
    int *hbad = reinterpret_cast<int *>(h_flags);  // pinned: the checks' verdict comes back asynchronously
    {  // element arrays: the raw CSR goes up once and the device places every
       // element (SELL slots, row-contiguous copy, split rows) together with
       // its FP32 screen copy
        const size_t n_sell = (size_t)std::max<long long>(sell_elems, 1);
        const size_t n_x = (size_t)std::max<long long>(x_elems, 1);
        const size_t n_l = (size_t)std::max<long long>(lnnz, 1);
        int *sc, *xc, *lc;
        double *xv, *lv;
        float *sa, *la;
        // the arrays with padding slots first: cleared together
        size_t cleared = 0;
        if (!arena.carve({{(void **)&sc, sizeof(int) * n_sell},
                          {(void **)&sa, sizeof(float) * n_sell},
                          {(void **)&xc, sizeof(int) * n_x},
                          {(void **)&xv, sizeof(double) * n_x},
                          {(void **)&lc, sizeof(int) * n_l},
                          {(void **)&lv, sizeof(double) * n_l},
                          {(void **)&la, sizeof(float) * n_l}})) {
            set_error("device allocation failed (layout element arrays)");
            return GDP_ERROR;
        }
        cleared = (size_t)((unsigned char *)(xv + n_x) - (unsigned char *)sc);
        GDP_CUDA(cudaMemsetAsync(sc, 0, cleared, stream));
        int *dord, *dspl, *dls, *dbad;
        long long *dlrp, *dlb;
        const int no_bad[2] = {INT_MAX, INT_MAX};
        Uploads maps;
        Uploads &um = small ? ups1 : maps;  // a small problem's row maps stay with its other arrays
        um.add(dord, order, sizeof(int) * (size_t)ns);
        um.add(dspl, split_rows.data(), sizeof(int) * (size_t)n_lrows);
        um.add(dlrp, lrow_ptr.data(), sizeof(long long) * ((size_t)n_lrows + 1));
        um.add(dls, len_start.data(), sizeof(int) * len_start.size());
        um.add(dlb, len_base.data(), sizeof(long long) * len_base.size());
        um.add(dbad, no_bad, sizeof(no_bad));
        if (small) {
            ups1.add(dcol, col, sizeof(int) * (size_t)nnz);
            ups1.add(dval, val, sizeof(double) * (size_t)nnz);
            ups1.add(drp, row_ptr, sizeof(int) * ((size_t)m + 1));
            ups1.add(dlhs, lhs, sizeof(double) * (size_t)m);
            ups1.add(drhs, rhs, sizeof(double) * (size_t)m);
        }
        const size_t sent = ups1.total;
        if (!ups1.send(arena, stream, stage, HostResources::kStageBytes)) {
            set_error("device allocation or upload failed (layout)");
            return GDP_ERROR;
        }
        if (stage) stage += std::min(sent, HostResources::kStageBytes);
        if (small) {
            GDP_CUDA(build_marking_counts(dcol, nnz, n, vp, vcur, vscan, stream));
        } else {
            uploader.t.join();
            stamps.mark(3);
            if (!up_err.empty()) {
                set_error(up_err);
                return GDP_ERROR;
            }
            GDP_CUDA(cudaStreamWaitEvent(stream, res->uploaded, 0));
            stamps.record(2, stream);
            if (!maps.send(tmp, stream, nullptr, 0)) {
                set_error("device allocation or upload failed (row maps)");
                return GDP_ERROR;
            }
        }
        GDP_CUDA(check_csr_elements(dcol, dval, nnz, n, dbad, 8 * n_sms, stream));
        LayoutBuild L;
        L.col = dcol; L.row_ptr = drp; L.val = dval;
        L.n_srows = ns; L.order = dord; L.pos_slice = P.pos_slice; L.slice_row0 = P.slice_row0;
        L.slice_lg = P.slice_lg; L.xptr = P.xptr; L.slice_ptr = P.slice_ptr;
        L.sell_col = sc; L.xcol = xc; L.xval = xv; L.sell_a32 = sa;
        L.g1_begin = g1_begin; L.la32 = la;
        L.n_lrows = n_lrows; L.split_rows = dspl; L.lrow_ptr = dlrp; L.lcol = lc; L.lval = lv;
        L.lhs = dlhs; L.rhs = drhs; L.len_start = dls; L.len_base = dlb; L.n_slices = n_slices;
        L.srow_len_out = d_srow_len; L.xptr_out = d_xptr; L.pos_slice_out = d_pos_slice;
        L.srow_lhs_out = d_srow_lhs; L.srow_rhs_out = d_srow_rhs;
        L.idx_cursor = vcur; L.var_ent = vent; L.n = n;
        // the layout build uses columns as indices only for the marking
        // index, which skips columns out of range, so it runs before the
        // element checks' verdict is read
        GDP_CUDA(build_layout_positions(L, 8 * n_sms, stream));
        GDP_CUDA(build_layout_elements(L, 8 * n_sms, stream));
        stamps.record(3, stream);
        stamps.mark(4);
        GDP_CUDA(cudaMemcpyAsync(hbad, dbad, sizeof(int) * 2, cudaMemcpyDeviceToHost, stream));
        P.sell_col = sc; P.sell_a32 = sa;
        P.xcol = xc; P.xval = xv;
        P.lcol = lc; P.lval = lv; P.la32 = la;
    }
    vec_blocks = std::max(1, std::min((std::max(n, std::max(ns + n_lrows, 1)) + 255) / 256, 8 * n_sms));
    // the marking index (also used by node batches when this context's rounds
    // never mark) was filled with the layout
    P.var_ptr = vp;
    P.var_ent = vent;
    // row-side infeasibility names a position's original row: the split rows
    // follow the SELL positions (the row order uploaded above is staged already)
    std::copy(split_rows.begin(), split_rows.end(), pos_row.begin() + ns);
    if (ns + n_lrows == 0) pos_row[0] = 0;
    ups2.add(P.pos_row, pos_row.data(), sizeof(int) * (size_t)std::max(ns + n_lrows, 1));
    std::vector<int> mtiles;
    for (int r = 0; r < n_lrows; r++)
        if (lrow_tile0[r + 1] - lrow_tile0[r] > 1)
            for (int t = lrow_tile0[r]; t < lrow_tile0[r + 1]; t++) mtiles.push_back(t);
    P.n_mtiles = (int)mtiles.size();
    if (mtiles.empty()) mtiles.push_back(0);
    ups2.add(P.mtiles, mtiles.data(), sizeof(int) * mtiles.size());
    P.n_items = (int)items.size();
    if (items.empty()) items.push_back(0);
    ups2.add(P.items, items.data(), sizeof(int) * items.size());
    P.use_marking = opts.use_marking < 0 ? 1 : (opts.use_marking > 2 ? 2 : opts.use_marking);
    // adaptive marking: mark when a round tightened fewer bounds than 1/16 of the variables
    P.mark_threshold = (unsigned)std::max(1, n / 16);
    RawVec<unsigned char> is_cont((size_t)std::max(n, 1));
    is_cont[0] = 0;
#pragma omp parallel for schedule(static) num_threads(host_threads_for(n))
    for (int j = 0; j < n; j++) is_cont[j] = vartype[j] == GDP_CONTINUOUS ? 1 : 0;
    ups2.add(P.is_cont, is_cont.data(), is_cont.size());
#undef GDP_UP
    // the rest goes up on the helper's stream while the device builds
    if (!ups2.send(arena, small ? stream : ups.s, stage,
                   stage ? (size_t)((unsigned char *)res->pinned + HostResources::kFlagBytes +
                                    HostResources::kStageBytes - stage)
                         : 0)) {
        set_error("device allocation or upload failed (work lists)");
        return GDP_ERROR;
    }
    const int npos = std::max(ns + n_lrows, 1);
    const int n_words = (n + 31) / 32;
    // deferred exact pass: per-class row queues (classes are contiguous position ranges)
    for (int c = 0; c < 6; c++) { P.cls_begin[c] = 0; P.cls_end[c] = 0; }
    for (int sl = n_slices - 1; sl >= 0; sl--) P.cls_begin[slice_lg[sl]] = slice_row0[sl];
    for (int sl = 0; sl < n_slices; sl++) P.cls_end[slice_lg[sl]] = slice_row0[sl + 1];
    P.n_chg_words = n_words;
    P.max_rounds = opts.max_rounds;
    P.spin_limit = opts.barrier_wait_kcycles > 0 ? 1000LL * opts.barrier_wait_kcycles : 4000000000LL;
    const size_t nl = (size_t)n_lrows, nt = (size_t)n_tiles, nv = (size_t)n;
    if (!arena.carve({{(void **)&P.tile_part, sizeof(TilePart) * nt},
                      {(void **)&P.tile_scr, sizeof(TileScr) * nt},
                      {(void **)&P.xrow, sizeof(XRow) * (size_t)ns},
                      {(void **)&P.xctr, sizeof(unsigned) * 32},
                      {(void **)&P.row_exact, sizeof(int) * nl},
                      {(void **)&P.lrow_margin, sizeof(double) * nl},
                      {(void **)&P.lrow_drift, sizeof(double) * nl},
                      {(void **)&P.lrow_skip, sizeof(int) * nl},
                      {(void **)&P.mark, sizeof(int) * (size_t)npos},
                      {(void **)&P.bnd, sizeof(double2) * nv},
                      {(void **)&P.bnd_nxt, sizeof(double2) * nv},
                      {(void **)&P.bnd32, sizeof(BndScr) * nv},  // stamped records
                      {(void **)&P.chg, sizeof(unsigned) * (size_t)n_words},
                      {(void **)&P.flags, sizeof(RoundFlags) * 3},
                      {(void **)&P.barrier, sizeof(unsigned) * 2},
                      {(void **)&P.queue, sizeof(unsigned) * 8}})) {
        set_error("device allocation failed");
        return GDP_ERROR;
    }
    if (!host_direct && alloc_staging() != GDP_OKAY) return GDP_ERROR;

    if (set_schedule(opts.sync_type, opts.ctas_per_sm, opts.cta_threads) != GDP_OKAY) return GDP_ERROR;
    stamps.mark(5);
    if (ups.s) GDP_CUDA(cudaStreamSynchronize(ups.s));
    GDP_CUDA(cudaStreamSynchronize(stream));  // before the raw CSR is freed and the verdict is read
    stamps.mark(6);
    stamps.report();
    raw.release();
    return element_error(hbad);
}

// Grid sizes of the loop drivers for the schedule (the layout is untouched).
// cta_threads 0: the default, 256, or one CTA of 512 threads for up to
// kOneCtaSlices slices of one-lane rows: its barrier is __syncthreads and its
// L1 stays valid from round to round (400 rows: 0.38 ms against 0.57 on 4 CTAs
// of 256 threads; 800 rows, 25 slices: 0.61 against 0.60). Its 16 warps also commit
// every round, a word of the change bitmap per warp and step, so the variables count
// too, the more the fewer warps the slices leave idle. MEGAKERNEL, one CTA against the
// grid: 30 rows, 125 words 0.062 and 0.071 ms, 375 words 0.080 and 0.072; 100 rows, 32
// words 0.082 and 0.086, 125 words 0.104 and 0.098; 400 rows, 10 words 0.29 and 0.34, 63
// words 0.43 and 0.38, 31,250 words 10.9 and 0.46.
constexpr int kOneCtaSlices = 16;
constexpr long long kOneCtaWords = 192;  // slices x words
// Warps that share a slice in place, up to 4 while that takes no more than
// kPartWarps warps: each screens the whole slice and runs its share of the exact
// rows, with more lanes per chain (30 rows: 0.089 -> 0.069 ms, 2,000 0.318 ->
// 0.299, 5,000 0.242 -> 0.226; 30,000 rows on 1,876 warps 0.411 -> 0.419).
constexpr int kMaxParts = 4, kPartWarps = 1024;
GDP_RETCODE Context::set_schedule(int sync_type, int ctas_per_sm, int cta_threads) {
    if (sync_type < CPU_LOOP || sync_type > MEGAKERNEL) {
        set_error("Unknown sync type");
        return GDP_ERROR;
    }
    if (cta_threads != 0 && cta_threads != 128 && cta_threads != 256 && cta_threads != 512) {
        set_error("cta_threads must be 128, 256 or 512");
        return GDP_ERROR;
    }
    GDP_CUDA(cudaSetDevice(opts.device));
    const bool one_lane = n_lrows == 0 && P.cls_end[0] == n_srows && P.cls_begin[0] == 0;
    const bool one_cta = cta_threads == 0 && one_lane && P.n_items <= kOneCtaSlices &&
                         (long long)P.n_items * P.n_chg_words <= kOneCtaWords;
    if (cta_threads == 0) cta_threads = one_cta ? 512 : 256;
    const int warps = cta_threads / 32;
    int act_bps = 0, cand_bps = 0, mega_bps = 0;
    // one-lane rows alone, and at most three slices per warp (16 warps per SM, fewer
    // with a limit): the exact pass in place. Megakernel, 130,000 rows of 2 to 16:
    // 0.86 ms in place, 1.04 queued; 200,000 0.99 and 1.06; 300,000 1.34 and 1.345;
    // 600,000 2.21 and 2.04
    P.in_place = one_lane && P.n_items <= n_sms * 3 * (ctas_per_sm > 0 ? std::min(16, ctas_per_sm * warps) : 16);
    GDP_CUDA(phase_occupancy(&act_bps, &cand_bps, &mega_bps, warps, P.in_place != 0));
    if (ctas_per_sm > 0) {
        act_bps = std::min(act_bps, ctas_per_sm);
        cand_bps = std::min(cand_bps, ctas_per_sm);
        mega_bps = std::min(mega_bps, ctas_per_sm);
    }
    // no more CTAs than a phase has work for a warp each: screen items, exact
    // items (a slice's rows make up to two), quarters of exact tiles, words of
    // the change bitmap. A grid barrier takes 1.6 us with 456 CTAs, 0.7 with 8.
    const long long cand_work = std::max(2LL * P.n_items, 4LL * P.n_mtiles);
    auto ctas_for = [](long long work, int w, int most) {
        return (int)std::max(1LL, std::min<long long>(most, (work + w - 1) / w));
    };
    act_blocks = ctas_for(P.n_items, kWarpsPerCta, act_bps * n_sms);
    cand_blocks = ctas_for(cand_work, kWarpsPerCta, cand_bps * n_sms);  // the exact-rows phase shares this launch
    P.parts = 1;
    if (P.in_place) {
        const long long most =
                one_cta ? warps : std::min<long long>((long long)std::max(1, mega_bps) * n_sms * warps, kPartWarps);
        while (P.parts < kMaxParts && 2LL * P.parts * P.n_items <= most) P.parts *= 2;
    }
    const long long mega_work = std::max({cand_work, (long long)P.n_chg_words, (long long)P.parts * P.n_items});
    mega_grid = one_cta ? 1 : ctas_for(mega_work, warps, std::max(1, mega_bps) * n_sms);
    mega_warps = warps;
    if (graph_exec && (opts.ctas_per_sm != ctas_per_sm)) {  // the GPU_LOOP graph holds the old grids
        cudaGraphExecDestroy(graph_exec);
        cudaGraphDestroy(graph);
        graph_exec = nullptr;
        graph = nullptr;
    }
    opts.sync_type = sync_type;
    opts.ctas_per_sm = ctas_per_sm;
    opts.cta_threads = one_cta ? 0 : cta_threads;  // what makes the same schedule again: 512 would make several CTAs
    return GDP_OKAY;
}

void Context::release_host_resources() {
    give_resources(res);
    res = nullptr;
    stream = nullptr;
    ev0 = ev1 = nullptr;
    h_flags = nullptr;
}

Context::~Context() {
    if (stream) cudaStreamSynchronize(stream);
    if (graph_exec) cudaGraphExecDestroy(graph_exec);
    if (graph) cudaGraphDestroy(graph);
    give_resources(res);
}

// ---- drivers ---------------------------------------------------------------
// CPU_LOOP: the host launches each round, one cooperative launch of the round
// loop per round, and reads its outcome from host memory that the launch
// writes. One round is queued ahead while the host waits for the one before
// (after the last round it does nothing), so the GPU does not wait for the
// host: 100 us a round with five launches, a copy and a synchronisation became
// 83 us on 60,001 power-law rows, 44 us became 27 us on 2,000 rows (with today's
// kernels 55 and 19).
GDP_RETCODE Context::rounds_cpu_loop(cudaStream_t s, int *launches, const std::function<void()> &meanwhile) {
    DevProblem Q = P;
    Q.spin_limit = kLongSpinLimit;  // a driver of launches: no wait of its rounds is an error to the caller
    volatile int *mail = reinterpret_cast<volatile int *>(h_flags + 2);
    mail[0] = 0;
    mail[1] = 1;
    int queued = 0;
    for (int round = 1; round <= opts.max_rounds; round++) {
        for (; queued < std::min(round + 1, opts.max_rounds); queued++)
            GDP_CUDA(launch_megakernel(Q, queued + 1, queued + 1, const_cast<int *>(mail), mega_grid, mega_warps, s));
        if (round == 1) meanwhile();
        // the round's mail, or an idle stream: the bounds were infeasible from
        // the start, or a launch ended with an error
        cudaError_t e = cudaErrorNotReady;
        for (int spin = 1; mail[0] < round && e == cudaErrorNotReady; spin++)
            if (spin % 256 == 0) e = cudaStreamQuery(s);
        if (e != cudaErrorNotReady) GDP_CUDA(e);
        if (mail[0] < round) break;
        // the device wrote mail[1] before mail[0]; an Arm host may read them the other way round
        std::atomic_thread_fence(std::memory_order_acquire);
        if (!mail[1]) break;
    }
    *launches += queued;
    return GDP_OKAY;
}

// GPU_LOOP: one CUDA graph whose conditional WHILE node repeats the round's
// phase kernels until the finalize kernel clears its condition -- the device-driven
// loop the reference built with dynamic parallelism (src/kernels/atomic_kernel.cuh:452-503).
GDP_RETCODE Context::build_graph() {
    struct Graph {  // destroyed unless it is complete
        cudaGraph_t g = nullptr;
        ~Graph() {
            if (g) cudaGraphDestroy(g);
        }
    } made;
    GDP_CUDA(cudaGraphCreate(&made.g, 0));
    cudaGraphConditionalHandle h;
    GDP_CUDA(cudaGraphConditionalHandleCreate(&h, made.g, 1u, cudaGraphCondAssignDefault));
    // cudaGraphNodeParams has no usable default constructor in C++: zero a raw buffer
    alignas(cudaGraphNodeParams) unsigned char cp_buf[sizeof(cudaGraphNodeParams)];
    std::memset(cp_buf, 0, sizeof(cp_buf));
    cudaGraphNodeParams &cp = *reinterpret_cast<cudaGraphNodeParams *>(cp_buf);
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    GDP_CUDA(cudaGraphAddNode(&node, made.g, nullptr, nullptr, 0, &cp));
    Sequence body(cp.conditional.phGraph_out[0]);
    GDP_CUDA(add_round(P, (unsigned long long)h, act_blocks, cand_blocks, vec_blocks, body));
    GDP_CUDA(cudaGraphInstantiate(&graph_exec, made.g, 0));
    graph = made.g;
    made.g = nullptr;
    return GDP_OKAY;
}

GDP_RETCODE Context::rounds_gpu_loop(cudaStream_t s) {
    if (!graph_exec && build_graph() != GDP_OKAY) return GDP_ERROR;
    GDP_CUDA(launch_round_begin(P, s));
    GDP_CUDA(cudaGraphLaunch(graph_exec, s));
    return GDP_OKAY;
}

// MEGAKERNEL: every round in one persistent cooperative launch.
GDP_RETCODE Context::rounds_megakernel(cudaStream_t s, int *launches) {
    GDP_CUDA(launch_megakernel(P, 1, opts.max_rounds, nullptr, mega_grid, mega_warps, s));
    *launches += 1;
    return GDP_OKAY;
}

GDP_RETCODE Context::run(const double *lb_in, const double *ub_in, double *lb_out, double *ub_out,
                         cudaStream_t s, gdp_stats *st) {
    P.max_rounds = opts.max_rounds;
    certified = false;
    // a call that fails leaves nothing of it running: its kernels use the caller's
    // arrays and the words that a later CPU_LOOP call reads its rounds from
    struct Drain {
        cudaStream_t s;
        bool on;
        ~Drain() {
            if (on) cudaStreamSynchronize(s);
        }
    } drain{s, true};
    GDP_CUDA(launch_start(P, lb_in, ub_in, vec_blocks, s));
    int launches = vec_blocks <= 32 ? 1 : 2;
    GDP_CUDA(cudaEventRecord(ev0, s));
    // The last kernel writes the result to the caller's arrays. The GPU's first
    // write to a page that nothing has touched yet is a fault of many microseconds
    // (new 8 MB arrays: 6 ms), so the host fills them with the inputs while the rounds
    // run, before that kernel is launched.
    const auto fill_outputs = [&] {
        if (lb_out != lb_in || ub_out != ub_in) copy_bounds(lb_in, ub_in, lb_out, ub_out);
    };
    const bool cpu_loop = !P.learned && opts.sync_type != MEGAKERNEL && opts.sync_type != GPU_LOOP;
    GDP_RETCODE rc;
    if (P.learned) rc = rounds_learned(s, &launches);
    else if (opts.sync_type == MEGAKERNEL) rc = rounds_megakernel(s, &launches);
    else if (opts.sync_type == GPU_LOOP) rc = rounds_gpu_loop(s);
    else rc = rounds_cpu_loop(s, &launches, fill_outputs);
    if (rc != GDP_OKAY) return rc;
    GDP_CUDA(cudaEventRecord(ev1, s));
    if (!cpu_loop) fill_outputs();
    GDP_CUDA(launch_finish(P, lb_out, ub_out, vec_blocks, s));
    launches++;
    GDP_CUDA(cudaMemcpyAsync(h_flags, P.flags, sizeof(RoundFlags), cudaMemcpyDeviceToHost, s));
    GDP_CUDA(cudaStreamSynchronize(s));
    drain.on = false;
    if (!P.learned && opts.sync_type == GPU_LOOP)
        launches += std::max(h_flags[0].rounds, 1) * (2 + (P.n_items > 0) + (P.n_mtiles > 0)) + 1;
    const RoundFlags &f = h_flags[0];
    if (f.error != kErrNone) {
        set_error("device error " + std::to_string(f.error) + " (grid barrier wait exceeded its limit)");
        if (st) st->device_error = f.error;
        return GDP_ERROR;
    }
    // P.bnd now holds a fixpoint certified by a round that changed nothing
    certified = !f.infeasible && !f.change;
    if (st) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, ev0, ev1) != cudaSuccess) {
            ms = -1.f;
            cudaGetLastError();
        }
        st->rounds = f.rounds;
        st->infeasible = f.infeasible;
        st->infeasible_var = (f.infeasible && f.infeasible_var != INT_MAX) ? f.infeasible_var : -1;
        st->infeasible_row = (f.infeasible && f.infeasible_row != INT_MAX) ? f.infeasible_row : -1;
        st->converged = (f.infeasible || !f.change) ? 1 : 0;
        st->device_error = f.error;
        st->kernel_launches = launches;
        st->changed_vars = (long long)f.changed_vars;
        st->rows_processed = (long long)f.rows_proc;
        st->nnz_processed = (long long)f.nnz_proc;
        st->nnz_exact = (long long)f.nnz_exact;
        st->rows_deferred = (long long)f.rows_deferred;
        st->divisions = (long long)f.divisions;
        st->rows_exact = (long long)f.rows_exact;
        st->rows_go = (long long)f.rows_go;
        st->rows_seqmax = (long long)f.rows_seqmax;
        st->rows_drift = (long long)f.rows_drift;
        st->nnz_drift = (long long)f.nnz_drift;
        st->full_rounds = f.full_rounds;
        // the rows read: without those left unread on their drift bound
        st->bytes_algorithmic = 12.0 * (double)(f.nnz_proc - f.nnz_drift) + 20.0 * (double)(f.rows_proc - f.rows_drift) +
                                36.0 * n * (double)f.rounds;
        st->device_ms = ms;
    }
    return GDP_OKAY;
}

// Learned marking: every round in one launch of the learned round loop.
GDP_RETCODE Context::rounds_learned(cudaStream_t s, int *launches) {
    GDP_CUDA((cudaError_t)launch_learned(P, learned_grid, vec_blocks, s));
    *launches += 2;
    return GDP_OKAY;
}

GDP_RETCODE Context::alloc_learned_state() {
    if (P.dirty) return GDP_OKAY;
    const size_t ns = (size_t)std::max(P.n_srows, 1);
    P.dirty = (int *)arena.alloc_bytes(sizeof(int) * ns);
    P.dcount = (int *)arena.alloc_bytes(sizeof(int) * ns);
    P.last_proc = (int *)arena.alloc_bytes(sizeof(int) * ns);
    P.last_tight = (int *)arena.alloc_bytes(sizeof(int) * ns);
    P.rstat = (float2 *)arena.alloc_bytes(sizeof(float2) * ns);
    P.rinfo = (unsigned *)arena.alloc_bytes(sizeof(unsigned) * ns);
    P.trace_n = (unsigned *)arena.alloc_bytes(sizeof(unsigned));
    if (!P.dirty || !P.dcount || !P.last_proc || !P.last_tight || !P.rstat || !P.rinfo || !P.trace_n) {
        set_error("device allocation failed (learned marking state)");
        return GDP_ERROR;
    }
    int bps = 0;
    GDP_CUDA((cudaError_t)learned_occupancy(&bps));
    learned_grid = std::max(1, bps) * n_sms;
    return GDP_OKAY;
}

GDP_RETCODE Context::set_model(const Mlp *m, float threshold, int min_len) {
    if (!m) {
        P.learned = 0;
        return GDP_OKAY;
    }
    if (alloc_learned_state() != GDP_OKAY) return GDP_ERROR;
    P.mlp = m->dev();
    P.tau = threshold;
    P.learn_min_len = std::max(0, min_len);
    P.learned = 1;
    return GDP_OKAY;
}

GDP_RETCODE Context::trace(double *lbs, double *ubs, int capacity, float *x_out, float *y_out, int *n_out,
                           gdp_stats *st) {
    if (capacity < 0 || (capacity > 0 && (!x_out || !y_out)) || !n_out) {
        set_error("bad trace arguments");
        return GDP_ERROR;
    }
    if (alloc_learned_state() != GDP_OKAY) return GDP_ERROR;
    const size_t cap = (size_t)std::max(capacity, 1);
    float *dx = nullptr, *dy = nullptr;
    GDP_CUDA(cudaMalloc(&dx, sizeof(float) * 16 * cap));
    GDP_CUDA(cudaMalloc(&dy, sizeof(float) * cap));
    const int saved = P.learned;
    P.learned = 2;
    P.trace_x = dx;
    P.trace_y = dy;
    P.trace_cap = (unsigned)capacity;
    GDP_RETCODE rc = GDP_OKAY;
    if (cudaMemsetAsync(P.trace_n, 0, sizeof(unsigned), stream) != cudaSuccess) rc = GDP_ERROR;
    if (rc == GDP_OKAY) rc = propagate_host(lbs, ubs, lbs, ubs, st);
    P.learned = saved;
    P.trace_x = nullptr;
    P.trace_y = nullptr;
    P.trace_cap = 0;
    unsigned cnt = 0;
    if (rc == GDP_OKAY) {
        if (cudaMemcpy(&cnt, P.trace_n, sizeof(unsigned), cudaMemcpyDeviceToHost) != cudaSuccess) rc = GDP_ERROR;
        const unsigned keep = std::min(cnt, (unsigned)capacity);
        if (rc == GDP_OKAY && keep) {
            if (cudaMemcpy(x_out, dx, sizeof(float) * 16 * keep, cudaMemcpyDeviceToHost) != cudaSuccess ||
                cudaMemcpy(y_out, dy, sizeof(float) * keep, cudaMemcpyDeviceToHost) != cudaSuccess)
                rc = GDP_ERROR;
        }
        *n_out = (int)keep;
        if (rc != GDP_OKAY) set_error("trace download failed");
    }
    cudaFree(dx);
    cudaFree(dy);
    return rc;
}

// Device copies of host bounds: for contexts without coherent access, and on
// first use for arrays that are not aligned as the kernels' loads need.
GDP_RETCODE Context::alloc_staging() {
    const size_t bytes = sizeof(double) * (size_t)std::max(n, 1);
    if (d_lb || arena.carve({{(void **)&d_lb, bytes}, {(void **)&d_ub, bytes}})) return GDP_OKAY;
    set_error("device allocation failed (bounds)");
    return GDP_ERROR;
}

GDP_RETCODE Context::propagate_host(const double *lbs_in, const double *ubs_in, double *lbs_out, double *ubs_out,
                                    gdp_stats *st) {
    bool aligned = true;
    for (const double *a : {lbs_in, ubs_in, (const double *)lbs_out, (const double *)ubs_out})
        aligned = aligned && reinterpret_cast<uintptr_t>(a) % sizeof(double) == 0;
    if (host_direct && aligned) {
        // coherent access to pageable memory (NVLink-C2C on Grace hosts): the
        // first kernel reads the caller's bounds where they are, and the last
        // one writes the result to them once the rounds succeeded
        const GDP_RETCODE rc = run(lbs_in, ubs_in, lbs_out, ubs_out, stream, st);
        if (rc != GDP_OKAY) copy_bounds(lbs_in, ubs_in, lbs_out, ubs_out);
        return rc;
    }
    copy_bounds(lbs_in, ubs_in, lbs_out, ubs_out);
    if (alloc_staging() != GDP_OKAY) return GDP_ERROR;
    const size_t bytes = sizeof(double) * (size_t)n;
    GDP_CUDA(cudaMemcpyAsync(d_lb, lbs_in, bytes, cudaMemcpyHostToDevice, stream));
    GDP_CUDA(cudaMemcpyAsync(d_ub, ubs_in, bytes, cudaMemcpyHostToDevice, stream));
    if (run(d_lb, d_ub, d_lb, d_ub, stream, st) != GDP_OKAY) return GDP_ERROR;
    GDP_CUDA(cudaMemcpyAsync(lbs_out, d_lb, bytes, cudaMemcpyDeviceToHost, stream));
    GDP_CUDA(cudaMemcpyAsync(ubs_out, d_ub, bytes, cudaMemcpyDeviceToHost, stream));
    GDP_CUDA(cudaStreamSynchronize(stream));
    return GDP_OKAY;
}

// The input bounds into the output arrays (a failed call leaves its input
// there), in chunks on the host threads: one thread copies a few GB/s.
void Context::copy_bounds(const double *lbs_in, const double *ubs_in, double *lbs_out, double *ubs_out) const {
    const long long chunk = 1 << 16, chunks = (n + chunk - 1) / chunk;
#pragma omp parallel for schedule(static) num_threads(host_threads_for(n))
    for (long long c = 0; c < chunks; c++) {
        const long long b = c * chunk, len = std::min(chunk, n - b);
        if (lbs_out != lbs_in) std::memcpy(lbs_out + b, lbs_in + b, sizeof(double) * (size_t)len);
        if (ubs_out != ubs_in) std::memcpy(ubs_out + b, ubs_in + b, sizeof(double) * (size_t)len);
    }
}

GDP_RETCODE Context::propagate_device(double *d_lbs, double *d_ubs, cudaStream_t s, gdp_stats *st) {
    if (!s) {
        // Handle 0 is the default stream to whoever fills the bounds (a framework's
        // current stream): what it has queued there so far comes first. The context's
        // stream does not wait for it by itself. While a stream that the default
        // stream waits for is being captured, the default stream takes no work.
        s = stream;
        cudaStreamCaptureStatus status;
        if (cudaStreamIsCapturing(cudaStreamLegacy, &status) == cudaSuccess) {
            GDP_CUDA(cudaEventRecord(res->uploaded, cudaStreamLegacy));
            GDP_CUDA(cudaStreamWaitEvent(s, res->uploaded, 0));
        } else {
            cudaGetLastError();
        }
    }
    return run(d_lbs, d_ubs, d_lbs, d_ubs, s, st);
}

}  // namespace gdp
