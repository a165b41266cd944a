// Zero-tile masks of device matrices (the layout is described with tile_mask_words in
// spmv_kernel.cuh).  One warp per 256 rows of a diagonal, a byte of each plane's word: 16-byte loads
// (all of them in flight at once), a ballot per load.  Reads every stored value once: 654 MB of the
// 20-qubit chain in 161 us (4.1 TB/s).  A batch of 24 small chains takes its masks at every run, where
// latency counts: 2 steps in 1,890 us against 1,997 with a whole 1,024-row word per warp.
#include <algorithm>
#include <vector>

#include "spmv_kernel.cuh"

namespace diaq_gb300 {

constexpr int kMaskWarps = 8;
constexpr int kMaskRows = 256;   // rows per warp: 8 tiles

// Byte `at` of each plane of the mask of one matrix (words = W * nd words per plane), by one warp.
template <typename T>
__device__ __forceinline__ void tile_mask_byte(const DiagMeta *__restrict__ meta, int64_t words, const T *__restrict__ re,
                                               const T *__restrict__ im, int64_t W, uint32_t *__restrict__ mask,
                                               int *__restrict__ has_im, int64_t at) {
    constexpr int V = VecOf<T>::V;            // rows per lane and load: a warp's load covers V tiles
    constexpr int N = kMaskRows / (32 * V);   // loads per plane
    constexpr int L = 32 / V;                 // lanes per tile
    constexpr uint32_t G = (1u << L) - 1u;
    const int lane = (int)threadIdx.x & 31;
    const int64_t j = (at >> 2) / W, r0 = ((at >> 2) - j * W) * 1024 + (at & 3) * kMaskRows;
    const DiagMeta m = meta[j];
    uint32_t br = 0u, bi = 0u;
    if (r0 >= m.lo && r0 + kMaskRows <= m.hi) {
        const T *pr = re + m.base + r0 + lane * V, *pi = im + m.base + r0 + lane * V;
        T a[N][V], b[N][V];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            load_vec_stream<T, V>(a[i], pr + i * 32 * V);
            load_vec_stream<T, V>(b[i], pi + i * 32 * V);
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            bool na = false, nb = false;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                na |= a[i][v] != (T)0;
                nb |= b[i][v] != (T)0;
            }
            const uint32_t ba = __ballot_sync(0xffffffffu, na), bb = __ballot_sync(0xffffffffu, nb);
#pragma unroll
            for (int t = 0; t < V; ++t) {
                if ((ba >> (t * L)) & G) br |= 1u << (i * V + t);
                if ((bb >> (t * L)) & G) bi |= 1u << (i * V + t);
            }
        }
    } else if (r0 < m.hi && r0 + kMaskRows > m.lo) {   // the diagonal's first or last rows
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const int64_t r = r0 + t * 32 + lane;
            const bool in = r >= m.lo && r < m.hi;
            const bool na = in && re[m.base + r] != (T)0, nb = in && im[m.base + r] != (T)0;
            if (__ballot_sync(0xffffffffu, na)) br |= 1u << t;
            if (__ballot_sync(0xffffffffu, nb)) bi |= 1u << t;
        }
    }
    // byte `at & 3` of the word, in memory order (little-endian)
    if (lane < 3) reinterpret_cast<uint8_t *>(mask)[lane * 4 * words + at] = (uint8_t)(lane == 0 ? br | bi : lane == 1 ? br : bi);
    if (has_im && bi && lane == 0) *has_im = 1;   // every writer stores 1
}

template <typename T>
__global__ void __launch_bounds__(kMaskWarps * 32)
    tile_mask_kernel(const DiagMeta *__restrict__ meta, int64_t words, const T *__restrict__ re,
                     const T *__restrict__ im, int64_t W, uint32_t *__restrict__ mask, int *__restrict__ has_im) {
    const int64_t at = (int64_t)blockIdx.x * kMaskWarps + (threadIdx.x >> 5);
    if (at < 4 * words) tile_mask_byte<T>(meta, words, re, im, W, mask, has_im, at);
}

// Many matrices at once: warp w works on byte w - first of the job whose bytes hold it.
template <typename T>
__global__ void __launch_bounds__(kMaskWarps * 32) tile_masks_kernel(const MaskJob *__restrict__ jobs, int n, int64_t bytes) {
    const int64_t w = (int64_t)blockIdx.x * kMaskWarps + (threadIdx.x >> 5);
    if (w >= bytes) return;
    int a = 0, b = n - 1;   // the last job that starts at or before w
    while (a < b) {
        const int m = (a + b + 1) >> 1;
        if (jobs[m].first <= w) a = m;
        else b = m - 1;
    }
    const MaskJob J = jobs[a];
    tile_mask_byte<T>(J.meta, J.words, (const T *)J.re, (const T *)J.im, J.W, J.mask, J.has_im, w - J.first);
}

int build_tile_mask(const Matrix &A, uint32_t *mask, cudaStream_t s, int *has_im) {
    if (A.nd == 0 || A.rows == 0) return DIAQ_OK;
    const int64_t W = tile_mask_words(A.rows), words = W * A.nd, blocks = (4 * words + kMaskWarps - 1) / kMaskWarps;
    if (blocks > 0x7fffffffll) return set_error(DIAQ_ERR_UNSUPPORTED, "tile mask: too many rows");
    // float pairs: the hi planes (the first `capacity` floats); a zero hi part has a zero lo part
    if (A.prec == DIAQ_C64 || A.prec == DIAQ_C128F2)
        tile_mask_kernel<float><<<(unsigned)blocks, kMaskWarps * 32, 0, s>>>(A.d_meta, words, (const float *)A.re,
                                                                             (const float *)A.im, W, mask, has_im);
    else
        tile_mask_kernel<double><<<(unsigned)blocks, kMaskWarps * 32, 0, s>>>(A.d_meta, words, (const double *)A.re,
                                                                              (const double *)A.im, W, mask, has_im);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

MaskJob mask_job(const Matrix &A, uint32_t *mask, int *has_im, int64_t first) {
    const int64_t W = tile_mask_words(A.rows);
    return MaskJob{A.d_meta, A.re, A.im, W, W * A.nd, mask, has_im, first};
}

int build_tile_masks(const MaskJob *jobs, int n, int64_t bytes, int prec, cudaStream_t s) {
    if (n == 0 || bytes == 0) return DIAQ_OK;
    const int64_t blocks = (bytes + kMaskWarps - 1) / kMaskWarps;
    if (blocks > 0x7fffffffll) return set_error(DIAQ_ERR_UNSUPPORTED, "tile mask: too many rows");
    if (prec == DIAQ_C64 || prec == DIAQ_C128F2)
        tile_masks_kernel<float><<<(unsigned)blocks, kMaskWarps * 32, 0, s>>>(jobs, n, bytes);
    else
        tile_masks_kernel<double><<<(unsigned)blocks, kMaskWarps * 32, 0, s>>>(jobs, n, bytes);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

const uint32_t *existing_tile_mask(const Matrix &A, cudaStream_t s) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return nullptr;
    }
    return A.tmask_ok ? A.tmask : nullptr;
}

const uint32_t *cached_tile_mask(const Matrix &A, cudaStream_t s) {
    if (A.nd == 0 || A.rows == 0 || !A.tmask) return nullptr;
    // no mask in a recorded graph: a replay could outlive the values the mask was taken from
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return nullptr;
    }
    if (A.tmask_ok) return A.tmask;
    // (an internal matrix is used on its own stream only: nobody waits)
    if (A.prec != DIAQ_C128F2) {
        if (build_tile_mask(A, A.tmask, s) != DIAQ_OK || (!A.internal && cudaStreamSynchronize(s) != cudaSuccess)) {
            cudaGetLastError();
            return nullptr;
        }
    } else {
        // is it real?  The flag sits behind the mask, zero since allocate(); it is only ever set, so
        // threads that make this call at the same time agree
        int *flag = (int *)(A.tmask + tile_mask_bytes(A.nd, A.rows) / sizeof(uint32_t)), has_im = 1;
        if (build_tile_mask(A, A.tmask, s, flag) != DIAQ_OK ||
            cudaMemcpyAsync(&has_im, flag, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        A.real = has_im == 0;
    }
    A.tmask_ok = true;
    return A.tmask;
}

}  // namespace diaq_gb300

using namespace diaq_gb300;

extern "C" int diaq_matrix_live_values(diaq_matrix_t A, int64_t *out, void *stream) {
    if (!A || !out) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    *out = 0;
    if (A->nd == 0 || A->rows == 0) return DIAQ_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t W = tile_mask_words(A->rows);
    uint32_t *mask = nullptr;
    DQ_CUDA(dev_malloc(&mask, tile_mask_bytes(A->nd, A->rows)));
    std::vector<uint32_t> h((size_t)A->nd * (size_t)W);
    int st = build_tile_mask(*A, mask, s);
    cudaError_t e = cudaSuccess;
    if (st == DIAQ_OK) e = cudaMemcpyAsync(h.data(), mask, sizeof(uint32_t) * h.size(), cudaMemcpyDeviceToHost, s);
    if (st == DIAQ_OK && e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(mask);
    if (st != DIAQ_OK) return st;
    if (e != cudaSuccess) return cuda_status(e, "live values", __FILE__, __LINE__);
    // every set bit is a 32-row tile with a nonzero: count its stored rows (a tile at either end
    // of a diagonal holds fewer)
    int64_t live = 0;
    for (int j = 0; j < A->nd; ++j) {
        const DiagMeta &m = A->meta[j];
        for (int64_t w = 0; w < W; ++w) {
            uint32_t bits = h[(size_t)j * W + w];
            while (bits) {
                const int b = __builtin_ctz(bits);
                bits &= bits - 1;
                const int64_t r0 = (w * 32 + b) * 32, r1 = r0 + 32;
                live += std::max<int64_t>(0, std::min(r1, m.hi) - std::max(r0, m.lo));
            }
        }
    }
    *out = live;
    return DIAQ_OK;
}

