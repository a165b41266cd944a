// C = A B with A in the row-aligned DIA format and B, C dense, all arrays already on the device:
// the reference's spmm_dia_device (src/spMM_device_gpu.cu:44-127, bound at
// include/pythonWrappers.cpp:622-633).
//
// Format: offsets int64[n_diags]; vals[k * n_rows + r] = A[r, r + offsets[k]] (entries whose
// column falls outside [0, n_cols) are ignored); B is n_cols x n_right and C n_rows x n_right,
// both row-major; float64 or interleaved complex128.  C is overwritten; diagonals are summed in
// the order given (duplicates add).
//
// Work split: thread e computes C's element e = r * n_right + j, so a warp's stores to C and its
// loads of B (at e + offset * n_right) are contiguous whatever n_right is, and the lanes of one
// row share the diagonal value (an L1 broadcast).  FP64 issue bounds it (4 multiply-adds per complex
// value), so a warp first finds the diagonals that reach its rows -- 32 at a time, a lane per diagonal,
// one ballot -- and takes only those, in the order given, the loads of kUnroll of them issued before the
// multiply-adds of the first.  Multiplying the entries outside the matrix by zero instead cost as
// much as the entries inside when offsets spread over the whole range: 65,536 x 16, 33 diagonals, complex
// 224 us that way, 123 now (97 % of the FP64 rate); real 63.5 and 37.9.
#include <algorithm>
#include <type_traits>

#include "diaq_internal.cuh"

namespace diaq_gb300 {

namespace {

constexpr int kSpmmThreads = 256;
constexpr int kUnroll = 4;

struct Real {
    using V = double;
    static __device__ __forceinline__ V zero() { return 0.0; }
    static __device__ __forceinline__ V mac(V acc, V a, V b) { return fma(a, b, acc); }
};

struct Cplx {
    using V = double2;
    static __device__ __forceinline__ V zero() { return make_double2(0.0, 0.0); }
    static __device__ __forceinline__ V mac(V acc, V a, V b) {
        acc.x = fma(-a.y, b.y, fma(a.x, b.x, acc.x));
        acc.y = fma(a.y, b.x, fma(a.x, b.y, acc.y));
        return acc;
    }
};

// I: the type of element, row and column numbers: with few diagonals the division by n_right and the
// shuffles are most of a warp's instructions.  And a grid-stride loop over some waves of blocks, as
// starting a block per 256 elements costs as much there.  10^6 x 64 complex elements, 1, 2 and 3
// diagonals: 700, 1,086 and 1,448 us with 64-bit numbers and a block per 256 elements, 539, 891 and 1,282 this way (every
// diagonal visited, no ballots: 554, 917, 1,329); real, 3 diagonals 706, 617 (885).  Blocks per SM: 64, which
// holds 100,000 x 20 in one wave of the loop (8 diagonals 61 us; 63 with 16); 16 for one or two diagonals
// (3 10^6 x 1 complex, 2 diagonals 51.5 us; 55 with 64).
template <class T, class I>
__global__ void __launch_bounds__(kSpmmThreads)
    spmm_dia_kernel(const int64_t *__restrict__ offsets, int nd, const typename T::V *__restrict__ vals,
                    int64_t M, int64_t K, const typename T::V *__restrict__ B, int64_t R,
                    typename T::V *__restrict__ C) {
    using V = typename T::V;
    const int lane = (int)threadIdx.x & 31;
    const int64_t total = M * R;
    const int64_t stride = (int64_t)gridDim.x * kSpmmThreads;
    for (int64_t e0 = (int64_t)blockIdx.x * kSpmmThreads + (threadIdx.x - lane); e0 < total; e0 += stride) {
        const I e = (I)e0 + lane, r = min(e, (I)(total - 1)) / (I)R;   // (lanes past the end load nothing)
        const I r0 = __shfl_sync(0xffffffffu, r, 0), r1 = __shfl_sync(0xffffffffu, r, 31);
        V acc = T::zero();
        for (int c0 = 0; c0 < nd; c0 += 32) {
            const int64_t own = c0 + lane < nd ? offsets[c0 + lane] : 0;
            uint32_t live = __ballot_sync(0xffffffffu, c0 + lane < nd && r1 + own >= 0 && r0 + own < K);
            // the diagonal of the lowest bit of live
            auto load = [&](V &a, V &b) {
                const int j = __ffs(live) - 1;
                live &= live - 1u;
                const I o = __shfl_sync(0xffffffffu, (I)own, j), c = r + o;   // (that of a live diagonal fits)
                const bool ok = e < (I)total && c >= 0 && c < (I)K;
                a = ok ? vals[(int64_t)(c0 + j) * M + r] : T::zero();
                b = ok ? __ldg(B + e + (int64_t)o * R) : T::zero();
            };
            while (__popc(live) >= kUnroll) {
                V a[kUnroll], b[kUnroll];
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) load(a[u], b[u]);
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) acc = T::mac(acc, a[u], b[u]);
            }
            while (live) {
                V a, b;
                load(a, b);
                acc = T::mac(acc, a, b);
            }
        }
        if (e < (I)total) C[e] = acc;
    }
}

}  // namespace

}  // namespace diaq_gb300

using namespace diaq_gb300;

extern "C" int diaq_spmm_dia_device(const int64_t *offsets, const void *vals, int n_diags, int64_t n_rows,
                                    int64_t n_cols, const void *B, int64_t n_right, void *C, int is_complex,
                                    void *stream) {
    if (n_diags < 0 || n_rows < 0 || n_cols < 0 || n_right < 0)
        return set_error(DIAQ_ERR_INVALID, "spmm_dia_device: sizes must be non-negative");
    if (n_rows == 0 || n_right == 0) return DIAQ_OK;
    if (!C || (n_diags > 0 && (!offsets || !vals || (n_cols > 0 && !B))))
        return set_error(DIAQ_ERR_INVALID, "spmm_dia_device: NULL array");
    const int64_t total = n_rows * n_right;
    const int64_t want = (total + kSpmmThreads - 1) / kSpmmThreads;
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, (n_diags <= 2 ? 16 : 64) * (int64_t)num_sms()));
    const cudaStream_t s = (cudaStream_t)stream;
    auto go = [&](auto kernel, auto *c) {
        using V = std::remove_pointer_t<decltype(c)>;
        kernel<<<grid, kSpmmThreads, 0, s>>>(offsets, n_diags, (const V *)vals, n_rows, n_cols, (const V *)B, n_right, c);
    };
    // 32 bits hold every element, row and column number, and a row plus the offset of a diagonal that
    // reaches it
    const bool narrow = total <= 0x7fffffffll && n_cols <= 0x7fffffffll - n_rows;
    if (is_complex) narrow ? go(spmm_dia_kernel<Cplx, int>, (double2 *)C) : go(spmm_dia_kernel<Cplx, int64_t>, (double2 *)C);
    else narrow ? go(spmm_dia_kernel<Real, int>, (double *)C) : go(spmm_dia_kernel<Real, int64_t>, (double *)C);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}
