// Device matrices: layout, allocation, upload/download, copy, precision conversion, prune.
// Replaces deviceDiaQMatrix (src/deviceMatrix_gpu.hpp:37-68, src/deviceMatrix_gpu.cu:30-113)
// and diaQMatrix::pruneMatrix (src/diaQMatrix.hpp:1543-1604).
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_set>

#include "diaq_internal.cuh"

namespace diaq_gb300 {

// ---- error state ---------------------------------------------------------------------------
static thread_local std::string g_last_error;

int set_error(int status, const std::string &msg) {
    g_last_error = msg;
    return status;
}

int cuda_status(cudaError_t e, const char *what, const char *file, int line) {
    const char *base = std::strrchr(file, '/');
    char buf[512];
    std::snprintf(buf, sizeof(buf), "CUDA error: %s (%s:%d) in %s", cudaGetErrorString(e),
                  base ? base + 1 : file, line, what);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();  // clear the sticky-free allocation error
        return set_error(DIAQ_ERR_OOM, buf);
    }
    return set_error(DIAQ_ERR_CUDA, buf);
}

size_t alloc_limit() {
    const char *v = std::getenv("DIAQ_DEVICE_ALLOC_LIMIT");
    if (!v || !*v) return SIZE_MAX;
    char *end = nullptr;
    const unsigned long long n = std::strtoull(v, &end, 10);
    return (end && *end == '\0') ? (size_t)n : SIZE_MAX;
}

// ---- memory pools ------------------------------------------------------------------------------
// One per device, made on first use and kept until the process exits.  `s` is a stream of its own for
// freeing memory that nothing uses any more: no order with anyone else's work is implied.
struct Block {
    void *p;
    size_t bytes;
    cudaEvent_t last;   // after the work that still uses it; NULL: none does
};
struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t s = nullptr;
    int64_t matrices = 0;        // alive on the device
    std::vector<Block> blocks;   // freed value arrays kept for reuse, oldest first
    size_t block_bytes = 0;
};
constexpr int kMaxDevices = 64;
static std::mutex g_pool_mu;
static DevicePool g_pools[kMaxDevices];

static cudaError_t pool_of(int dev, DevicePool **out) {   // g_pool_mu held, dev current
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    DevicePool &P = g_pools[dev];
    *out = &P;
    if (P.pool) return cudaSuccess;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = kPoolKeep - P.block_bytes;
    e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e == cudaSuccess && !P.s) e = cudaStreamCreateWithFlags(&P.s, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        cudaMemPoolDestroy(pool);
        return e;
    }
    P.pool = pool;
    return cudaSuccess;
}

cudaError_t pool_malloc(void **p, size_t bytes, cudaStream_t s) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        DevicePool *P = nullptr;
        e = pool_of(dev, &P);
        if (e != cudaSuccess) return e;
        pool = P->pool;
    }
    return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

void pool_free_idle(void *p, int device) {
    cudaStream_t s = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        if (device >= 0 && device < kMaxDevices) s = g_pools[device].s;
    }
    if (p) cudaFreeAsync(p, s);
}

// Value arrays of kBlockMin bytes and more are cudaMalloc's, and up to kBlockKeep bytes of freed ones are
// kept per device for arrays of the same size.  The driver's pool grows by 0.75 ms and shrinks by 1.3 ms
// per GB where cudaMalloc and cudaFree take 0.25 and 0.6, so whatever it had not kept cost more than with
// plain allocations.  With cudaMalloc alone, with the pool alone, and this way: making and destroying a
// 20-qubit chain, the only matrix, 0.9, 1.7 and 0.8 ms; chain, H H of 18 qubits and both destroyed 5.7, 7.6
// and 4.9 ms; pruned H H of 20 qubits (12 GB) 32, 44 and 28 ms; H H of 18 qubits again and again 4.2, 1.6 and
// 1.6 ms.  Below kBlockMin the pool's cheap suballocation counts for more (small products and exponentials).
// And cudaFree gives a kept array back at once, whatever still reads it.
static size_t block_size(size_t bytes) { return (bytes + kBlockGrain - 1) / kBlockGrain * kBlockGrain; }

// `by` bytes more kept as blocks (g_pool_mu held): the driver's pool may keep the rest of kPoolKeep.
static void count_block(DevicePool &P, int64_t by) {
    P.block_bytes += by;
    uint64_t keep = kPoolKeep - P.block_bytes;
    if (P.pool) cudaMemPoolSetAttribute(P.pool, cudaMemPoolAttrReleaseThreshold, &keep);
}

static void free_blocks(std::vector<Block> &v) {
    for (const Block &b : v) {
        if (cudaFree(b.p) != cudaSuccess) cudaGetLastError();   // (refused during a capture: stays allocated)
        if (b.last) cudaEventDestroy(b.last);
    }
    v.clear();
}

// Whether value arrays of this size come from the driver's pool.  result: those of a product that goes to
// the caller as it is.  Programs make these again and again, and where they are too large to be kept here
// the pool holds on to them until something synchronises (unpruned H H of 20 qubits, 11 GB: 8.4 ms a
// product, 11.0 from cudaMalloc; the first one, with its matrix made and destroyed, 34 and 18).
static bool array_pooled(size_t bytes, int device, bool result) {
    if (bytes < kBlockMin || device < 0 || device >= kMaxDevices) return true;
    return result && bytes > kBlockKeep / 2;   // (a matrix has two arrays)
}

// A value array on the current device; work on s may use it.
static cudaError_t array_malloc(void **p, size_t bytes, int device, cudaStream_t s, bool pooled) {
    if (pooled) return dev_malloc_async(p, bytes, s);
    if (bytes > alloc_limit()) return cudaErrorMemoryAllocation;
    const size_t size = block_size(bytes);
    Block got{nullptr, 0, nullptr};
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        DevicePool &P = g_pools[device];
        for (size_t i = P.blocks.size(); i-- > 0;)
            if (P.blocks[i].bytes == size) {
                got = P.blocks[i];
                P.blocks.erase(P.blocks.begin() + i);
                count_block(P, -(int64_t)size);
                break;
            }
    }
    cudaError_t e = cudaSuccess;
    if (!got.p) {
        e = cudaMalloc(p, size);
        return alloc_failed(e) ? cudaMalloc(p, size) : e;
    }
    if (got.last) {
        e = cudaStreamWaitEvent(s, got.last, 0);
        cudaEventDestroy(got.last);
    }
    if (e != cudaSuccess) {
        cudaFree(got.p);
        return e;
    }
    *p = got.p;
    return cudaSuccess;
}

// Gives back a value array of the device.  idle: nothing uses it any more; else work on s may.
static void array_free(void *p, size_t bytes, int device, cudaStream_t s, bool idle, bool pooled) {
    if (!p) return;
    if (pooled) {
        if (idle) pool_free_idle(p, device);
        else cudaFreeAsync(p, s);
        return;
    }
    Block b{p, block_size(bytes), nullptr};
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    bool keep = b.bytes <= kBlockKeep / 2;
    if (keep && !idle)   // an event of a stream being captured marks no work
        keep = cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone &&
               cudaEventCreateWithFlags(&b.last, cudaEventDisableTiming) == cudaSuccess &&
               cudaEventRecord(b.last, s) == cudaSuccess;
    std::vector<Block> out;
    if (keep) {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        DevicePool &P = g_pools[device];
        while (P.block_bytes + b.bytes > kBlockKeep) {
            out.push_back(P.blocks.front());
            count_block(P, -(int64_t)P.blocks.front().bytes);
            P.blocks.erase(P.blocks.begin());
        }
        P.blocks.push_back(b);
        count_block(P, (int64_t)b.bytes);
    } else {
        out.push_back(b);
    }
    free_blocks(out);   // (waits for the device)
}

bool alloc_failed(cudaError_t e) {
    if (e != cudaErrorMemoryAllocation) return false;
    cudaGetLastError();
    std::vector<Block> out;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        for (auto &P : g_pools) {
            out.insert(out.end(), P.blocks.begin(), P.blocks.end());
            P.blocks.clear();
            count_block(P, -(int64_t)P.block_bytes);
        }
    }
    bool any = !out.empty();
    free_blocks(out);
    std::lock_guard<std::mutex> lock(g_pool_mu);
    for (auto &P : g_pools)
        if (P.pool) {
            uint64_t kept = 0, used = 0;
            cudaMemPoolGetAttribute(P.pool, cudaMemPoolAttrReservedMemCurrent, &kept);
            cudaMemPoolGetAttribute(P.pool, cudaMemPoolAttrUsedMemCurrent, &used);
            any = (cudaMemPoolTrimTo(P.pool, 0) == cudaSuccess && kept > used) || any;
        }
    return any;
}

// Counts the matrices alive on a device; when the last one goes, all but kPoolRest of what is kept is
// given back.
static void count_matrix(int device, int by) {
    if (device < 0 || device >= kMaxDevices) return;
    std::vector<Block> out;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        DevicePool &P = g_pools[device];
        P.matrices += by;
        if (P.matrices != 0) return;
        out.swap(P.blocks);
        count_block(P, -(int64_t)P.block_bytes);
        uint64_t kept = 0;
        if (P.pool && cudaMemPoolGetAttribute(P.pool, cudaMemPoolAttrReservedMemCurrent, &kept) == cudaSuccess &&
            kept > kPoolRest) {
            cudaStreamSynchronize(P.s);   // the frees have landed
            cudaMemPoolTrimTo(P.pool, kPoolRest);
        }
    }
    free_blocks(out);
}

int num_sms() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

// ---- geometry --------------------------------------------------------------------------------
int64_t diag_len(int64_t rows, int64_t cols, int64_t d) {
    // src/diaQMatrix.hpp:390-409 for offsets inside the matrix
    int64_t len;
    if (d < 0) len = rows + d;
    else if (d > 0) len = cols - d;
    else len = rows < cols ? rows : cols;
    if (len > rows) len = rows;
    else if (len > cols) len = cols;
    return len < 0 ? 0 : len;
}

int plan_layout(Matrix &M, int64_t rows, int64_t cols, int32_t nd, const int32_t *off) {
    if (rows < 0 || cols < 0) return set_error(DIAQ_ERR_INVALID, "matrix shape must be non-negative");
    // the kernels keep row indices, offsets and row ranges in 32 bits (the reference's are 32-bit too)
    if (rows >= ((int64_t)1 << 31) || cols >= ((int64_t)1 << 31))
        return set_error(DIAQ_ERR_UNSUPPORTED, "matrix dimensions must be below 2^31");
    if (nd < 0) return set_error(DIAQ_ERR_INVALID, "diagonal count must be non-negative");
    if (nd > 0 && !off) return set_error(DIAQ_ERR_INVALID, "offsets pointer is NULL");
    M.rows = rows;
    M.cols = cols;
    M.nd = nd;
    M.off.assign(off, off + nd);
    M.meta.resize(nd);
    const bool ascending = std::adjacent_find(off, off + nd, [](int32_t a, int32_t b) { return a >= b; }) == off + nd;
    std::unordered_set<int32_t> seen;   // (ascending offsets are distinct)
    if (!ascending) seen.reserve(nd * 2 + 1);
    int64_t cursor = kAlign, pstart = 0;
    for (int32_t k = 0; k < nd; ++k) {
        const int64_t d = off[k];
        if (d <= -rows || d >= cols)
            return set_error(DIAQ_ERR_INVALID, "diagonal offset " + std::to_string(d) +
                                                   " lies outside a " + std::to_string(rows) + " x " +
                                                   std::to_string(cols) + " matrix");
        if (!ascending && !seen.insert(off[k]).second)
            return set_error(DIAQ_ERR_INVALID, "diagonal offset " + std::to_string(d) + " appears twice");
        const int64_t len = diag_len(rows, cols, d);
        const int64_t lo = d < 0 ? -d : 0;
        const int64_t gap = ((lo - cursor) % kAlign + kAlign) % kAlign;
        const int64_t s = cursor + gap;  // s == lo (mod kAlign)
        DiagMeta &m = M.meta[k];
        m.base = s - lo;
        m.lo = lo;
        m.hi = lo + len;
        m.pstart = pstart;
        m.off = off[k];
        m.slot = k;
        m.pad = 0;
        cursor = s + len;
        pstart += len;
    }
    // a multiple of kAlign, so that a second plane (C128F2) starts aligned as well
    M.capacity = (cursor + 2 * kAlign - 1) / kAlign * kAlign;
    M.total = pstart;
    return DIAQ_OK;
}

// The metadata block: DiagMeta records and, behind them, the zero-tile mask's storage (and a flag: does
// the matrix hold an imaginary part), so that SpMV calls never allocate (it is filled on first use).
static size_t meta_bytes(const Matrix &M) { return (sizeof(DiagMeta) * (size_t)M.nd + 255) / 256 * 256; }

static size_t block_bytes(const Matrix &M) { return meta_bytes(M) + tile_mask_bytes(M.nd, M.rows) + sizeof(int); }

// The planes come from the pool.  A caller's matrix has its metadata block from cudaMalloc: freeing
// that waits for all work on the device (as freeing the planes so would), after which the planes may
// go back to the pool whatever streams the matrix was used on.
int allocate(Matrix &M, cudaStream_t s, bool zero) {
    cudaGetDevice(&M.device);
    const size_t bytes = (size_t)M.capacity * M.elem(), block = block_bytes(M);
    if (M.nd == 0 && !M.internal) {   // no metadata block: plain allocations
        DQ_CUDA(dev_malloc(&M.re, bytes));
        DQ_CUDA(dev_malloc(&M.im, bytes));
    } else {
        M.pooled = array_pooled(bytes, M.device, !zero && !M.internal);
        DQ_CUDA(array_malloc(&M.re, bytes, M.device, s, M.pooled));
        DQ_CUDA(array_malloc(&M.im, bytes, M.device, s, M.pooled));
    }
    if (zero) {
        DQ_CUDA(cudaMemsetAsync(M.re, 0, bytes, s));
        DQ_CUDA(cudaMemsetAsync(M.im, 0, bytes, s));
    }
    if (M.nd > 0) {
        if (M.internal)
            DQ_CUDA(dev_malloc_async(&M.d_meta, block, s));
        else
            DQ_CUDA(dev_malloc(&M.d_meta, block));
        M.tmask = (uint32_t *)((uint8_t *)M.d_meta + meta_bytes(M));
        DQ_CUDA(cudaMemsetAsync((uint8_t *)M.tmask + tile_mask_bytes(M.nd, M.rows), 0, sizeof(int), s));
        DQ_CUDA(cudaMemcpyAsync(M.d_meta, M.meta.data(), sizeof(DiagMeta) * M.nd, cudaMemcpyHostToDevice, s));
        // the host vector may be reallocated later; finish the copy before returning
        DQ_CUDA(cudaStreamSynchronize(s));
    }
    return DIAQ_OK;
}

int publish(Matrix &M) {
    if (!M.internal) return DIAQ_OK;
    const size_t block = block_bytes(M);
    DiagMeta *d = nullptr;
    void *re = nullptr, *im = nullptr;
    if (M.nd > 0) {
        DQ_CUDA(dev_malloc(&d, block));
    } else {   // as allocate() has it
        const size_t bytes = (size_t)M.capacity * M.elem();
        DQ_CUDA(dev_malloc(&re, bytes));
        cudaError_t e = dev_malloc(&im, bytes);
        if (e == cudaSuccess) e = cudaMemcpyAsync(re, M.re, bytes, cudaMemcpyDeviceToDevice, M.stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(im, M.im, bytes, cudaMemcpyDeviceToDevice, M.stream);
        if (e != cudaSuccess) {
            cudaFree(re);
            cudaFree(im);
            return cuda_status(e, "publish", __FILE__, __LINE__);
        }
    }
    cudaError_t e = cudaSuccess;
    if (d) e = cudaMemcpyAsync(d, M.d_meta, block, cudaMemcpyDeviceToDevice, M.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(M.stream);
    if (e != cudaSuccess) {
        cudaFree(d);
        cudaFree(re);
        cudaFree(im);
        return cuda_status(e, "publish", __FILE__, __LINE__);
    }
    if (d) {
        cudaFreeAsync(M.d_meta, M.stream);
        M.d_meta = d;
        M.tmask = (uint32_t *)((uint8_t *)d + meta_bytes(M));
    } else {
        array_free(M.re, (size_t)M.capacity * M.elem(), M.device, M.stream, false, M.pooled);
        array_free(M.im, (size_t)M.capacity * M.elem(), M.device, M.stream, false, M.pooled);
        M.re = re;
        M.im = im;
    }
    M.internal = false;
    return DIAQ_OK;
}

void release(Matrix &M) {
    const size_t bytes = (size_t)M.capacity * M.elem();
    if (M.internal) {
        array_free(M.re, bytes, M.device, M.stream, false, M.pooled);
        array_free(M.im, bytes, M.device, M.stream, false, M.pooled);
        if (M.d_meta) cudaFreeAsync(M.d_meta, M.stream);
    } else if (M.nd > 0) {
        // The planes go back only after a wait that succeeded: given back without one, the next
        // allocation could take them from under kernels still queued.  A cudaFree that is refused
        // (while a stream is being captured in global mode) has waited for nothing; the planes then
        // stay allocated, as the block itself does.
        // (a matrix whose allocation failed half-way was used by nothing but its own stream's fills)
        const cudaError_t e = M.d_meta ? cudaFree(M.d_meta) : cudaStreamSynchronize(M.stream);
        if (e == cudaSuccess) {
            array_free(M.re, bytes, M.device, nullptr, true, M.pooled);
            array_free(M.im, bytes, M.device, nullptr, true, M.pooled);
        } else {
            cudaGetLastError();   // not the next launch's
        }
    } else {
        cudaFree(M.re);
        cudaFree(M.im);
    }
    M.re = M.im = nullptr;
    M.d_meta = nullptr;
    M.tmask = nullptr;
    M.tmask_ok = false;
}

int make_zero(int64_t rows, int64_t cols, int32_t nd, const int32_t *off, int prec,
              cudaStream_t s, Matrix **out, bool zero, bool internal) {
    if (prec != DIAQ_C128 && prec != DIAQ_C64 && prec != DIAQ_C128F2)
        return set_error(DIAQ_ERR_INVALID, "precision must be DIAQ_C128, DIAQ_C64 or DIAQ_C128F2");
    Matrix *M = new diaq_matrix_s();
    cudaGetDevice(&M->device);
    count_matrix(M->device, 1);
    M->prec = prec;
    M->internal = internal;
    M->stream = s;
    int st = plan_layout(*M, rows, cols, nd, off);
    if (st == DIAQ_OK) st = allocate(*M, s, zero);
    if (st != DIAQ_OK) {
        destroy(M);
        return st;
    }
    *out = M;
    return DIAQ_OK;
}

// Block j zeroes gap j: [0, start of diagonal 0) for j = 0, [end of j - 1, start of j) between
// diagonals, [end of the last, capacity) for j = nd -- in each of the `planes` planes of
// `capacity` elements of size esz in re and im.
__global__ void zero_gaps_kernel(const DiagMeta *__restrict__ meta, int nd, int64_t capacity, int esz, int planes,
                                 unsigned char *re, unsigned char *im) {
    const int j = blockIdx.x;
    const int64_t a = j == 0 ? 0 : meta[j - 1].base + meta[j - 1].hi;
    const int64_t b = j == nd ? capacity : meta[j].base + meta[j].lo;
    for (int p = 0; p < planes; ++p)
        for (int64_t e = a + threadIdx.x; e < b; e += blockDim.x)
            for (int k = 0; k < esz; ++k) {
                re[(p * capacity + e) * esz + k] = 0;
                im[(p * capacity + e) * esz + k] = 0;
            }
}

int zero_gaps(const Matrix &M, cudaStream_t s) {
    const int planes = M.prec == DIAQ_C128F2 ? 2 : 1;
    const int esz = M.prec == DIAQ_C128 ? 8 : 4;
    zero_gaps_kernel<<<M.nd + 1, 64, 0, s>>>(M.d_meta, M.nd, M.capacity, esz, planes, (unsigned char *)M.re,
                                             (unsigned char *)M.im);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

void destroy(Matrix *M) {
    if (!M) return;
    release(*M);
    count_matrix(M->device, -1);
    delete static_cast<diaq_matrix_s *>(M);
}

// ---- copy kernels ------------------------------------------------------------------------------
// One y-row of the grid per diagonal (strided when there are more diagonals than grid rows),
// x over the diagonal's rows.

template <typename TS, typename TD>
__global__ void scatter_kernel(const DiagMeta *__restrict__ meta, int nd, const TS *__restrict__ sre,
                               const TS *__restrict__ sim, TD *__restrict__ dre,
                               TD *__restrict__ dim) {
    for (int k = blockIdx.y; k < nd; k += gridDim.y) {
        const DiagMeta m = meta[k];
        const int64_t len = m.hi - m.lo;
        for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < len;
             j += (int64_t)gridDim.x * blockDim.x) {
            dre[m.base + m.lo + j] = (TD)sre[m.pstart + j];
            dim[m.base + m.lo + j] = (TD)sim[m.pstart + j];
        }
    }
}

template <typename TS>
__global__ void gather_kernel(const DiagMeta *__restrict__ meta, int nd, const TS *__restrict__ sre,
                              const TS *__restrict__ sim, double *__restrict__ dre,
                              double *__restrict__ dim) {
    for (int k = blockIdx.y; k < nd; k += gridDim.y) {
        const DiagMeta m = meta[k];
        const int64_t len = m.hi - m.lo;
        for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < len;
             j += (int64_t)gridDim.x * blockDim.x) {
            dre[m.pstart + j] = (double)sre[m.base + m.lo + j];
            dim[m.pstart + j] = (double)sim[m.base + m.lo + j];
        }
    }
}

// dst diagonal k <- src diagonal map[k] (same offset, so same rows), with conversion.
template <typename TS, typename TD>
__global__ void remap_kernel(const DiagMeta *__restrict__ smeta, const TS *__restrict__ sre,
                             const TS *__restrict__ sim, const DiagMeta *__restrict__ dmeta,
                             TD *__restrict__ dre, TD *__restrict__ dim, const int32_t *__restrict__ map,
                             int nd) {
    for (int k = blockIdx.y; k < nd; k += gridDim.y) {
        const DiagMeta dm = dmeta[k];
        const DiagMeta sm = smeta[map ? map[k] : k];
        for (int64_t r = dm.lo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < dm.hi;
             r += (int64_t)gridDim.x * blockDim.x) {
            dre[dm.base + r] = (TD)sre[sm.base + r];
            dim[dm.base + r] = (TD)sim[sm.base + r];
        }
    }
}

// Per diagonal: does it hold a value other than exact zero?
template <typename T>
__global__ void nonzero_kernel(const DiagMeta *__restrict__ meta, int nd, const T *__restrict__ re,
                               const T *__restrict__ im, int32_t *__restrict__ flag) {
    for (int k = blockIdx.x; k < nd; k += gridDim.x) {
        const DiagMeta m = meta[k];
        int nz = 0;
        for (int64_t r = m.lo + threadIdx.x; r < m.hi && !nz; r += blockDim.x)
            nz = (re[m.base + r] != (T)0) || (im[m.base + r] != (T)0);
        nz = __syncthreads_or(nz);
        if (threadIdx.x == 0) flag[k] = nz;
    }
}

static dim3 diag_grid(const Matrix &M) {
    int64_t maxlen = 1;
    for (const auto &m : M.meta) maxlen = std::max(maxlen, m.hi - m.lo);
    int64_t gx = (maxlen + 1023) / 1024;
    gx = std::min<int64_t>(gx, 4 * num_sms());
    const int64_t gy = std::min<int64_t>(std::max<int32_t>(M.nd, 1), 65535);
    return dim3((unsigned)std::max<int64_t>(gx, 1), (unsigned)gy);
}

int scatter_packed(Matrix &M, const double *re, const double *im, cudaStream_t s) {
    M.tmask_ok = false;
    if (M.nd == 0 || M.total == 0) return DIAQ_OK;
    if (M.prec == DIAQ_C128F2) return f2_scatter(M, re, im, s);
    const dim3 g = diag_grid(M);
    if (M.prec == DIAQ_C128)
        scatter_kernel<double, double><<<g, 256, 0, s>>>(M.d_meta, M.nd, re, im, (double *)M.re, (double *)M.im);
    else
        scatter_kernel<double, float><<<g, 256, 0, s>>>(M.d_meta, M.nd, re, im, (float *)M.re, (float *)M.im);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

int gather_packed(const Matrix &M, double *re, double *im, cudaStream_t s) {
    if (M.nd == 0 || M.total == 0) return DIAQ_OK;
    if (M.prec == DIAQ_C128F2) return f2_gather(M, re, im, s);
    const dim3 g = diag_grid(M);
    if (M.prec == DIAQ_C128)
        gather_kernel<double><<<g, 256, 0, s>>>(M.d_meta, M.nd, (const double *)M.re, (const double *)M.im, re, im);
    else
        gather_kernel<float><<<g, 256, 0, s>>>(M.d_meta, M.nd, (const float *)M.re, (const float *)M.im, re, im);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

// Copy the values of src into dst (dst's offsets are a subset of src's; map[k] = src slot of
// dst slot k, NULL when the slots coincide).
static int remap(const Matrix &src, Matrix &dst, const int32_t *d_map, cudaStream_t s) {
    dst.tmask_ok = false;
    if (dst.nd == 0) return DIAQ_OK;
    const dim3 g = diag_grid(dst);
    if (src.prec == DIAQ_C128 && dst.prec == DIAQ_C128)
        remap_kernel<double, double><<<g, 256, 0, s>>>(src.d_meta, (const double *)src.re, (const double *)src.im,
                                                       dst.d_meta, (double *)dst.re, (double *)dst.im, d_map, dst.nd);
    else if (src.prec == DIAQ_C128 && dst.prec == DIAQ_C64)
        remap_kernel<double, float><<<g, 256, 0, s>>>(src.d_meta, (const double *)src.re, (const double *)src.im,
                                                      dst.d_meta, (float *)dst.re, (float *)dst.im, d_map, dst.nd);
    else if (src.prec == DIAQ_C64 && dst.prec == DIAQ_C128)
        remap_kernel<float, double><<<g, 256, 0, s>>>(src.d_meta, (const float *)src.re, (const float *)src.im,
                                                      dst.d_meta, (double *)dst.re, (double *)dst.im, d_map, dst.nd);
    else
        remap_kernel<float, float><<<g, 256, 0, s>>>(src.d_meta, (const float *)src.re, (const float *)src.im,
                                                     dst.d_meta, (float *)dst.re, (float *)dst.im, d_map, dst.nd);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

int copy_as(const Matrix &A, int prec, cudaStream_t s, Matrix **out, bool internal) {
    Matrix *C = nullptr;
    DQ_TRY(make_zero(A.rows, A.cols, A.nd, A.off.data(), prec, s, &C, true, internal));
    int st = DIAQ_OK;
    if (A.prec == DIAQ_C128F2 && prec == DIAQ_C128F2) {
        cudaError_t e = cudaMemcpyAsync(C->re, A.re, A.capacity * A.elem(), cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(C->im, A.im, A.capacity * A.elem(), cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) st = cuda_status(e, "copy", __FILE__, __LINE__);
    } else if (A.prec == DIAQ_C128F2 || prec == DIAQ_C128F2) {
        st = f2_convert(A, *C, s);
    } else {
        st = remap(A, *C, nullptr, s);
    }
    if (st == DIAQ_OK && !internal) {
        cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) st = cuda_status(e, "cudaStreamSynchronize", __FILE__, __LINE__);
    }
    if (st != DIAQ_OK) {
        destroy(C);
        return st;
    }
    *out = C;
    return DIAQ_OK;
}

// flag[k]: diagonal k of A holds a value other than exact zero.  Waits for s.
static int nonzero_diagonals(const Matrix &A, cudaStream_t s, std::vector<int32_t> &flag) {
    flag.assign((size_t)A.nd, 1);
    if (A.nd > 0) {
        int32_t *d_flag = nullptr;
        DQ_CUDA(dev_malloc_async(&d_flag, sizeof(int32_t) * A.nd, s));
        const int grid = (int)std::min<int64_t>(A.nd, 65535);
        if (A.prec == DIAQ_C128)
            nonzero_kernel<double><<<grid, 256, 0, s>>>(A.d_meta, A.nd, (const double *)A.re, (const double *)A.im, d_flag);
        else
            nonzero_kernel<float><<<grid, 256, 0, s>>>(A.d_meta, A.nd, (const float *)A.re, (const float *)A.im, d_flag);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(flag.data(), d_flag, sizeof(int32_t) * A.nd, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        cudaFreeAsync(d_flag, s);
        if (e != cudaSuccess) return cuda_status(e, "prune flags", __FILE__, __LINE__);
    }
    return DIAQ_OK;
}

static int keep_diagonals(const Matrix &A, const std::vector<int32_t> &flag, cudaStream_t s, Matrix **out, bool internal);

int prune_matrix(const Matrix &A, cudaStream_t s, Matrix **out) {
    if (A.prec == DIAQ_C128F2) return set_error(DIAQ_ERR_UNSUPPORTED, "prune: convert a c128f2 matrix to c128 first");
    std::vector<int32_t> flag;
    DQ_TRY(nonzero_diagonals(A, s, flag));
    return keep_diagonals(A, flag, s, out, false);
}

int prune_internal(Matrix **M, cudaStream_t s) {
    std::vector<int32_t> flag;
    DQ_TRY(nonzero_diagonals(**M, s, flag));
    if (std::find(flag.begin(), flag.end(), 0) == flag.end()) return DIAQ_OK;   // nothing to drop, nothing to copy
    Matrix *P = nullptr;
    DQ_TRY(keep_diagonals(**M, flag, s, &P, true));
    destroy(*M);
    *M = P;
    return DIAQ_OK;
}

static int keep_diagonals(const Matrix &A, const std::vector<int32_t> &flag, cudaStream_t s, Matrix **out, bool internal) {
    std::vector<int32_t> keep_off, map;
    for (int32_t k = 0; k < A.nd; ++k)
        if (flag[k]) {
            keep_off.push_back(A.off[k]);
            map.push_back(k);
        }
    Matrix *C = nullptr;
    DQ_TRY(make_zero(A.rows, A.cols, (int32_t)keep_off.size(), keep_off.data(), A.prec, s, &C, true, internal));
    int st = DIAQ_OK;
    if (C->nd > 0) {
        int32_t *d_map = nullptr;
        cudaError_t e = dev_malloc_async(&d_map, sizeof(int32_t) * C->nd, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(d_map, map.data(), sizeof(int32_t) * C->nd, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) st = remap(A, *C, d_map, s);
        else st = cuda_status(e, "prune map", __FILE__, __LINE__);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (d_map) cudaFreeAsync(d_map, s);
        if (st == DIAQ_OK && e != cudaSuccess) st = cuda_status(e, "prune copy", __FILE__, __LINE__);
    }
    if (st != DIAQ_OK) {
        destroy(C);
        return st;
    }
    *out = C;
    return DIAQ_OK;
}

}  // namespace diaq_gb300

// ---- C ABI -------------------------------------------------------------------------------------
using namespace diaq_gb300;

extern "C" {

const char *diaq_last_error(void) { return g_last_error.c_str(); }

const char *diaq_version(void) { return "diaq_gb300 0.1 (sm_103a)"; }

int diaq_matrix_create(int64_t rows, int64_t cols, int32_t ndiag, const int32_t *offsets,
                       const double *re, const double *im, int values_on_device, int precision,
                       void *stream, diaq_matrix_t *out) {
    if (!out) return set_error(DIAQ_ERR_INVALID, "out pointer is NULL");
    *out = nullptr;
    if ((re == nullptr) != (im == nullptr))
        return set_error(DIAQ_ERR_INVALID, "re and im must both be given or both be NULL");
    cudaStream_t s = (cudaStream_t)stream;
    Matrix *M = nullptr;
    DQ_TRY(make_zero(rows, cols, ndiag, offsets, precision, s, &M));
    if (re && M->total > 0) {
        const double *dre = re, *dim = im;
        double *stage = nullptr;
        int st = DIAQ_OK;
        if (!values_on_device) {
            const size_t bytes = sizeof(double) * (size_t)M->total;
            cudaError_t e = dev_malloc(&stage, 2 * bytes);
            if (e == cudaSuccess) e = cudaMemcpyAsync(stage, re, bytes, cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) e = cudaMemcpyAsync(stage + M->total, im, bytes, cudaMemcpyHostToDevice, s);
            if (e != cudaSuccess) st = cuda_status(e, "upload", __FILE__, __LINE__);
            dre = stage;
            dim = stage + M->total;
        }
        if (st == DIAQ_OK) st = scatter_packed(*M, dre, dim, s);
        if (st == DIAQ_OK) {
            cudaError_t e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) st = cuda_status(e, "cudaStreamSynchronize", __FILE__, __LINE__);
        }
        if (stage) cudaFree(stage);
        if (st != DIAQ_OK) {
            destroy(M);
            return st;
        }
    }
    *out = handle(M);
    return DIAQ_OK;
}

int diaq_matrix_destroy(diaq_matrix_t A) {
    destroy(A);
    return DIAQ_OK;
}

int diaq_matrix_info(diaq_matrix_t A, int64_t *rows, int64_t *cols, int32_t *ndiag,
                     int64_t *total, int *precision) {
    if (!A) return set_error(DIAQ_ERR_INVALID, "matrix handle is NULL");
    if (rows) *rows = A->rows;
    if (cols) *cols = A->cols;
    if (ndiag) *ndiag = A->nd;
    if (total) *total = A->total;
    if (precision) *precision = A->prec;
    return DIAQ_OK;
}

int diaq_matrix_offsets(diaq_matrix_t A, int32_t *offsets) {
    if (!A || (!offsets && A->nd > 0)) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    if (A->nd) std::memcpy(offsets, A->off.data(), sizeof(int32_t) * A->nd);
    return DIAQ_OK;
}

int diaq_matrix_download(diaq_matrix_t A, double *re, double *im, int dst_on_device, void *stream) {
    if (!A) return set_error(DIAQ_ERR_INVALID, "matrix handle is NULL");
    if (A->total == 0) return DIAQ_OK;
    if (!re || !im) return set_error(DIAQ_ERR_INVALID, "destination pointer is NULL");
    cudaStream_t s = (cudaStream_t)stream;
    if (dst_on_device) {
        DQ_TRY(gather_packed(*A, re, im, s));
        DQ_CUDA(cudaStreamSynchronize(s));
        return DIAQ_OK;
    }
    double *stage = nullptr;
    const size_t bytes = sizeof(double) * (size_t)A->total;
    DQ_CUDA(dev_malloc(&stage, 2 * bytes));
    int st = gather_packed(*A, stage, stage + A->total, s);
    cudaError_t e = cudaSuccess;
    if (st == DIAQ_OK) e = cudaMemcpyAsync(re, stage, bytes, cudaMemcpyDeviceToHost, s);
    if (st == DIAQ_OK && e == cudaSuccess) e = cudaMemcpyAsync(im, stage + A->total, bytes, cudaMemcpyDeviceToHost, s);
    if (st == DIAQ_OK && e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(stage);
    if (st == DIAQ_OK && e != cudaSuccess) st = cuda_status(e, "download", __FILE__, __LINE__);
    return st;
}

int diaq_matrix_copy(diaq_matrix_t A, void *stream, diaq_matrix_t *out) {
    if (!A || !out) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    Matrix *C = nullptr;
    DQ_TRY(copy_as(*A, A->prec, (cudaStream_t)stream, &C));
    *out = handle(C);
    return DIAQ_OK;
}

int diaq_matrix_convert(diaq_matrix_t A, int precision, void *stream, diaq_matrix_t *out) {
    if (!A || !out) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    Matrix *C = nullptr;
    DQ_TRY(copy_as(*A, precision, (cudaStream_t)stream, &C));
    *out = handle(C);
    return DIAQ_OK;
}

int diaq_matrix_prune(diaq_matrix_t A, void *stream, diaq_matrix_t *out) {
    if (!A || !out) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    Matrix *C = nullptr;
    DQ_TRY(prune_matrix(*A, (cudaStream_t)stream, &C));
    *out = handle(C);
    return DIAQ_OK;
}

}  // extern "C"
