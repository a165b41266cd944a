// The diagonal-sparse SpMV kernel (y = A x for up to K right-hand sides at once), shared by the
// plain SpMV entry points and the fused time-evolution terms, which differ only in the epilogue.
//
// Work split: thread t of block b owns the V consecutive rows r0 = (b*256 + t)*V .. r0+V-1: by default
// one row in float64, whose products are bound by FP64 issue, and 4 rows, one 16-byte vector, in float32
// (default_cfg); the evolution plans' launch shapes choose among 1, 2 and 4.  For every diagonal
// (metadata staged in shared memory in chunks), the thread loads the V matrix values of its rows as one
// aligned vector per array (the row-phase aligned layout makes base + r0 a multiple of V), so a warp
// streams 256 or 512 contiguous bytes per array per diagonal: fully coalesced.  x is read at
// columns r0+d .. r0+d+V-1 -- as one vector when d is a multiple of V, else element by element --
// through L1/L2, where the reuse across diagonals and neighbouring blocks lives (the state
// vector of a 2^20-row problem is 16 MB, L2-resident on GB300).  Each row's sum runs over the
// diagonals in slot order with fused multiply-adds; the epilogue functor gets the V sums per
// right-hand side.  Variants for few rows (dia_spmv_row_kernel, dia_spmv_split_kernel) and for several
// float32 states off the 16-byte boundaries (dia_spmv_strip_kernel) follow it.
#pragma once

#include "diaq_internal.cuh"

namespace diaq_gb300 {

constexpr int kSpmvThreads = 256;
constexpr int kMetaChunk = 256;

// ---- zero-tile mask --------------------------------------------------------------------------------
// One bit per diagonal and 32-row tile: bit t of word w of diagonal j is set when rows
// 32 (32 w + t) .. 32 (32 w + t) + 31 of diagonal j hold a nonzero value (real or imaginary part),
// word (j, w) at mask[j * tile_mask_words(rows) + w]; two further planes of nd * tile_mask_words(rows)
// words follow, the same for the real parts alone and for the imaginary parts alone.  Kernels whose warps cover aligned 32-row
// tiles skip a clear tile whole -- no matrix load, no state window, no multiply-adds.  In
// Pauli-sum Hamiltonians most off-diagonal tiles are zero: the hopping term of qubits k, k+1
// fills a quarter of the rows of its diagonal, in runs of 2^k rows.  Leaving out terms a * x
// with a == 0 changes no finite sum (up to the sign of a zero result).
//
// The plane words let a kernel go further in the tiles it visits: where one plane of the matrix is
// all zero (the Hamiltonians of real spin chains, and each Pauli string's diagonal, hold one plane
// only) it loads the other plane alone and runs two of the four multiply-adds of a complex product.
// What is left out, 0 * x, matters only for an infinite or NaN x -- and such an x also reaches one of
// the two sums through the plane that is used, since every value of a visited tile is multiplied.  So
// a row whose sums come out non-finite (from x, from stored values, or by overflow) is summed again
// with both planes: the results are those of the full product in every case.
// Fill the mask of A (tile_mask_bytes(A.nd, A.rows)) on stream s; *has_im (on the device, may be NULL)
// is set to 1 if A holds a nonzero imaginary part and else left as it is.
int build_tile_mask(const Matrix &A, uint32_t *mask, cudaStream_t s, int *has_im = nullptr);
// The masks of many matrices of one precision in one launch: jobs (on the device) in the order of
// `first`, the running sum of their mask_job_bytes; bytes is the whole sum.
struct MaskJob {
    const DiagMeta *meta;
    const void *re, *im;
    int64_t W, words;    // words per diagonal and per plane
    uint32_t *mask;
    int *has_im;
    int64_t first;
};
MaskJob mask_job(const Matrix &A, uint32_t *mask, int *has_im, int64_t first);
inline int64_t mask_job_bytes(const Matrix &A) { return 4 * tile_mask_words(A.rows) * A.nd; }
int build_tile_masks(const MaskJob *jobs, int n, int64_t bytes, int prec, cudaStream_t s);
// A's own mask, built (and waited for) on first use after its values were last written; NULL when
// it cannot be had now (s is being captured into a graph, or allocation failed): visit every tile.
const uint32_t *cached_tile_mask(const Matrix &A, cudaStream_t s);
// A's mask if it is built and current (never builds, never allocates), else NULL.
const uint32_t *existing_tile_mask(const Matrix &A, cudaStream_t s);

// VR consecutive values of T as one aligned vector load (VR * sizeof(T) bytes).
template <typename T, int VR>
struct Vec;
template <>
struct Vec<double, 2> {
    using type = double2;
};
template <>
struct Vec<double, 1> {
    using type = double;
};
template <>
struct Vec<float, 4> {
    using type = float4;
};
template <>
struct Vec<float, 2> {
    using type = float2;
};
template <>
struct Vec<float, 1> {
    using type = float;
};

// The widest vector: 16 bytes.
template <typename T>
struct VecOf {
    static constexpr int V = 16 / sizeof(T);
    using type = typename Vec<T, V>::type;
};

template <typename VT, typename T, int VR>
__device__ __forceinline__ void unpack(T (&dst)[VR], const VT &v) {
    if constexpr (VR == 1) {
        dst[0] = v;
    } else if constexpr (VR == 2) {
        dst[0] = v.x;
        dst[1] = v.y;
    } else {
        dst[0] = v.x;
        dst[1] = v.y;
        dst[2] = v.z;
        dst[3] = v.w;
    }
}

template <typename T, int VR = VecOf<T>::V>
__device__ __forceinline__ void load_vec(T (&dst)[VR], const T *p) {
    using VT = typename Vec<T, VR>::type;
    unpack<VT, T, VR>(dst, __ldg(reinterpret_cast<const VT *>(p)));
}

// A state value.  In a chained kernel (see launch_chained) a predecessor may still be writing the
// vector when the kernel starts, so the load is of the ordinary, coherent kind and the pointers to the
// vector are not __restrict__; elsewhere it is __ldg, which promises data that nobody writes while the
// kernel lives and is the faster one under load (24 chains batched: 1,225 us against 1,305; __ldca,
// opaque to the compiler's scheduling: 1,273).
template <bool CHAINED, typename T>
__device__ __forceinline__ T load_state(const T *p) {
    if constexpr (CHAINED) return *p;
    else return __ldg(p);
}

// Matrix values stream once: evict them first from L2, keeping x resident.
template <typename T, int VR = VecOf<T>::V>
__device__ __forceinline__ void load_vec_stream(T (&dst)[VR], const T *p) {
    using VT = typename Vec<T, VR>::type;
    unpack<VT, T, VR>(dst, __ldcs(reinterpret_cast<const VT *>(p)));
}

template <int BYTES>
__device__ __forceinline__ bool aligned_to(const void *p) {
    return (reinterpret_cast<uintptr_t>(p) & (uintptr_t)(BYTES - 1)) == 0;
}
__device__ __forceinline__ bool aligned16(const void *p) { return aligned_to<16>(p); }

// Asks L2 for the values one diagonal holds in a block's rows: one bulk prefetch per plane and
// run of live 32-row tiles among the block's tiles from row row0 (mask bits `bits`, bit j = tile
// j), clipped to the stored rows [lo, hi) widened to whole tiles.  Tile starts are 128-byte
// aligned in every plane (base is a multiple of 32 values), and the widened ends stay inside the
// allocation (a guard of 32 values before the first diagonal and after the last).  real: the real
// plane only.  The
// interleaved kernels (256 rows per block) use it; in the planar kernel below and the float-pair
// SpMV (1,024 rows per block, up to 8 KB per diagonal and plane ahead) it measured slower on the
// 20-qubit chain -- one-state Horner evolution 2,106 -> 1,693 states x steps/s, float-pair SpMV
// 99 -> 132 us -- and is not called there.  for_live_runs calls f(a, b) for each such run of rows.
template <class F>
__device__ __forceinline__ void for_live_runs(uint32_t bits, int64_t row0, int64_t lo, int64_t hi, F &&f) {
    while (bits) {
        const int j = __ffs(bits) - 1;
        const uint32_t run = bits >> j;
        const int len = run == 0xffffffffu ? 32 : __ffs(~run) - 1;   // live tiles j .. j + len - 1
        bits = len + j >= 32 ? 0u : bits & ~(((1u << len) - 1u) << j);
        const int64_t a = max(row0 + 32 * j, lo & ~(int64_t)31);
        const int64_t b = min(row0 + 32 * (int64_t)(j + len), (hi + 31) & ~(int64_t)31);
        if (a < b) f(a, b);
    }
}
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
template <typename T>
__device__ __forceinline__ void prefetch_tiles_l2(const T *are, const T *aim, bool real, int64_t base, int64_t lo,
                                                  int64_t hi, uint32_t bits, int64_t row0) {
    for_live_runs(bits, row0, lo, hi, [&](int64_t a, int64_t b) {
        const uint32_t bytes = (uint32_t)(b - a) * (uint32_t)sizeof(T);
        prefetch_l2(are + base + a, bytes);
        if (!real) prefetch_l2(aim + base + a, bytes);
    });
}

// Mask bits of the `tiles` (1 .. 32) tiles from row row0 in the 1024-row mask word w.
__device__ __forceinline__ uint32_t block_tile_bits(uint32_t w, int64_t row0, int tiles) {
    return tiles >= 32 ? w : (w >> ((row0 >> 5) & 31)) & ((1u << tiles) - 1u);
}

// Whether any of the sums is infinite or NaN, from their bit patterns.
__device__ __forceinline__ uint32_t abs_hi(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t abs_hi(double v) { return (uint32_t)__double2hiint(v) & 0x7fffffffu; }
template <typename T>
__device__ __forceinline__ bool any_nonfinite(uint32_t largest) {
    return largest >= (sizeof(T) == 4 ? 0x7f800000u : 0x7ff00000u);
}

// Whether sums taken by planes, whose largest and smallest abs_hi these are, have to be taken again in
// full: one is not finite -- unless all are NaN, which no further product changes (a vector that has
// overflowed turns to NaN within a product or two, and products with it need not cost twice: 205 -> 76 us
// for a NaN state on the 20-qubit chain in c128, as for a finite one).
template <typename T>
__device__ __forceinline__ bool unsettled(uint32_t largest, uint32_t smallest) {
    return any_nonfinite<T>(largest) && smallest <= (sizeof(T) == 4 ? 0x7f800000u : 0x7ff00000u);
}

// One diagonal's value base and the word of its imaginary plane's mask for the block's rows.
struct BaseIm {
    int64_t base;
    uint32_t im;
    uint32_t pad;
};

// One diagonal's (q = offset, lo, hi) products with rows r0 .. r0 + V - 1 of up to K states, the real
// (RE) and the imaginary (IM) plane of the matrix each taken or left out.
template <typename T, int K, int V, bool RE, bool IM, bool CHAINED>
__device__ __forceinline__ void dia_mac(const int4 &q, int64_t base, int64_t r0, const T *__restrict__ are,
                                        const T *__restrict__ aim, const T *xr, const T *xi,
                                        int64_t ldx, int kq, T (&accr)[K][V], T (&acci)[K][V]) {
    constexpr int VB = V * (int)sizeof(T);
    const int64_t lo = q.y, hi = q.z;
    const bool full = (r0 >= lo) && (r0 + V <= hi);
    T ar[V], ai[V];
    if constexpr (RE) load_vec_stream<T, V>(ar, are + base + r0);
    if constexpr (IM) load_vec_stream<T, V>(ai, aim + base + r0);
    if (!full) {
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (r0 + v < lo || r0 + v >= hi) ar[v] = ai[v] = (T)0;
    }
    const int64_t c = r0 + q.x;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (k >= kq) break;
        const T *pxr = xr + k * ldx + c;
        const T *pxi = xi + k * ldx + c;
        T xrv[V], xiv[V];
        if (full && aligned_to<VB>(pxr) && aligned_to<VB>(pxi)) {
            using VT = typename Vec<T, V>::type;
            unpack<VT, T, V>(xrv, load_state<CHAINED>(reinterpret_cast<const VT *>(pxr)));
            unpack<VT, T, V>(xiv, load_state<CHAINED>(reinterpret_cast<const VT *>(pxi)));
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const bool ok = (r0 + v >= lo) && (r0 + v < hi);
                xrv[v] = ok ? load_state<CHAINED>(pxr + v) : (T)0;
                xiv[v] = ok ? load_state<CHAINED>(pxi + v) : (T)0;
            }
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
            if constexpr (RE) accr[k][v] = fma(ar[v], xrv[v], accr[k][v]);
            if constexpr (IM) accr[k][v] = fma(-ai[v], xiv[v], accr[k][v]);
            if constexpr (RE) acci[k][v] = fma(ar[v], xiv[v], acci[k][v]);
            if constexpr (IM) acci[k][v] = fma(ai[v], xrv[v], acci[k][v]);
        }
    }
}

// nrhs states in nchunk chunks of up to K, VR rows per thread.  Block b works on chunk
// b % nchunk of row tile b / nchunk: the blocks of one row tile are neighbours in launch order and
// run at the same time, so the matrix tile they all read comes from HBM once and from L2 for the
// other chunks -- the matrix traffic of one launch over all states, with the registers of K.
//
// Four float32 rows a thread with two and four states are held to the registers of four and three blocks
// per SM.  Left alone, the choice of planes took the plans' instances past them (66-70 and 90
// registers): two Horner steps of 24 terms on two 19-qubit Ising states 2,338 us, 1,441 with 58 registers;
// 20 qubits 3,650 and 2,767.  The other shapes do best as the compiler has them.
template <typename T, int K, int VR>
constexpr int kSpmvMinBlocks = sizeof(T) == 4 && VR == 4 ? (K == 2 ? 4 : K == 4 ? 3 : 0) : 0;

template <typename T, int K, int VR, class Epi>
__global__ void __launch_bounds__(kSpmvThreads, kSpmvMinBlocks<T, K, VR>)
    dia_spmv_kernel(const DiagMeta *__restrict__ meta, int nd, const T *__restrict__ are,
                    const T *__restrict__ aim, int64_t rows, const T *xr,
                    const T *xi, int64_t ldx, int nrhs, int nchunk, const uint32_t *__restrict__ tmask,
                    int64_t mw, Epi epi0) {
    constexpr int V = VR;
    // per diagonal: offset, row range and the real plane's mask word of the block's rows in one
    // 16-byte record (rows < 2^31), the value base and the imaginary plane's word in another
    __shared__ int4 sq[kMetaChunk];
    __shared__ BaseIm sb[kMetaChunk];
    const int chunk = (int)(blockIdx.x % (unsigned)nchunk);
    const int64_t tile = blockIdx.x / (unsigned)nchunk;
    const int q0 = chunk * K;
    const int kq = min(K, nrhs - q0);
    xr += q0 * ldx;
    xi += q0 * ldx;
    const Epi epi = epi0.shifted(q0);
    const int64_t r0 = (tile * kSpmvThreads + threadIdx.x) * V;
    // a block's 256 V rows (V | 4) lie in one 1024-row mask word; a thread's V rows in one tile
    const int64_t mword = (tile * kSpmvThreads * V) >> 10;
    const int tbit = (int)((r0 >> 5) & 31);
    T accr[K][V], acci[K][V];

    if (Epi::kChained && nd == 0) dependency_wait();
    for (int pass = 0;; ++pass) {  // a second pass, with both planes, for rows that are not finite
#pragma unroll
        for (int q = 0; q < K; ++q)
#pragma unroll
            for (int v = 0; v < V; ++v) accr[q][v] = acci[q][v] = (T)0;
        for (int c0 = 0; c0 < nd; c0 += kMetaChunk) {
            const int cn = min(kMetaChunk, nd - c0);
            if (pass == 0 || nd > kMetaChunk) {
                __syncthreads();
                for (int i = threadIdx.x; i < cn; i += kSpmvThreads) {
                    const DiagMeta m = meta[c0 + i];
                    const int64_t w = (int64_t)(c0 + i) * mw + mword;
                    const uint32_t wr = tmask ? tmask[nd * mw + w] : 0xffffffffu;
                    const uint32_t wi = tmask ? tmask[2 * nd * mw + w] : 0xffffffffu;
                    sq[i] = make_int4(m.off, (int)m.lo, (int)m.hi, (int)wr);
                    sb[i] = BaseIm{m.base, wi, 0u};
                }
                __syncthreads();
                if constexpr (Epi::kChained) dependency_wait();
            }
            if (r0 >= rows) continue;
#pragma unroll 2
            for (int k = 0; k < cn; ++k) {
                const int4 q = sq[k];
                const BaseIm b = sb[k];
                const int64_t lo = q.y, hi = q.z;
                bool re = ((uint32_t)q.w >> tbit) & 1u, im = (b.im >> tbit) & 1u;
                if (r0 + V <= lo || r0 >= hi || !(re || im)) continue;
                if (pass) re = im = true;
                // whole bodies rather than conditions around the multiply-adds: those become
                // predicates, and a predicated-off FP64 multiply-add takes its issue slots all the same
                // (165 us per c128 product on the 20-qubit chain).  float32 takes imaginary-only tiles
                // as complex ones: a third body cost its complex tiles 4 %
                if (!im)
                    dia_mac<T, K, V, true, false, Epi::kChained>(q, b.base, r0, are, aim, xr, xi, ldx, kq, accr, acci);
                else if (re || sizeof(T) == 4)
                    dia_mac<T, K, V, true, true, Epi::kChained>(q, b.base, r0, are, aim, xr, xi, ldx, kq, accr, acci);
                else
                    dia_mac<T, K, V, false, true, Epi::kChained>(q, b.base, r0, are, aim, xr, xi, ldx, kq, accr, acci);
            }
        }
        if (pass || !tmask) break;
        uint32_t big = 0u, small = ~0u;
#pragma unroll
        for (int q = 0; q < K; ++q)
#pragma unroll
            for (int v = 0; v < V; ++v) {
                big = max(big, max(abs_hi(accr[q][v]), abs_hi(acci[q][v])));
                small = min(small, min(abs_hi(accr[q][v]), abs_hi(acci[q][v])));
            }
        // with several chunks the staging barriers make the second pass the whole block's
        const bool again = unsettled<T>(big, small);
        if (!(nd > kMetaChunk ? __syncthreads_or(again) : again)) break;
    }
    if constexpr (Epi::kChained) dependents_go();
    if (r0 < rows) epi.template apply<T, K, V>(r0, rows, kq, accr, acci);
}

// dia_spmv_kernel for float32, several states and windows off the 16-byte boundaries: a thread's V rows
// are 32 apart (row of lane l: strip + 32 v + l), so that a warp's loads are runs of 128 bytes whatever
// the offset of the diagonal and the alignment of the vectors, and the tiles of its strip are live or
// not for the whole warp.  With vectors of 4 rows an unaligned window falls apart into single loads 16
// bytes apart.  The sums are those of dia_spmv_kernel, in its order.  250,007-row band, 37 diagonals, 5
// states: 33.5 us against 39.9 (6 states of 300,000 rows, 30 diagonals: 31.1 against 41.5).  Bound by
// latency: three states (64 registers, 4 blocks per SM) read the matrix fewer times than two and leave
// a fuller last wave; two 37, four 51, five 61 us; 48 registers spill, 59.
constexpr int kStripStates = 3, kStripRows = 4;
template <int K, int V, class Epi>
__global__ void __launch_bounds__(kSpmvThreads)
    dia_spmv_strip_kernel(const DiagMeta *__restrict__ meta, int nd, const float *__restrict__ are,
                          const float *__restrict__ aim, int64_t rows, const float *__restrict__ xr, const float *__restrict__ xi, int64_t ldx,
                          int nrhs, int nchunk, const uint32_t *__restrict__ tmask, int64_t mw, Epi epi0) {
    static_assert(!Epi::kChained, "waits for no predecessor");
    __shared__ int4 sq[kMetaChunk];
    __shared__ BaseIm sb[kMetaChunk];
    const int chunk = (int)(blockIdx.x % (unsigned)nchunk);
    const int64_t tile = blockIdx.x / (unsigned)nchunk;
    const int q0 = chunk * K;
    const int kq = min(K, nrhs - q0);
    xr += q0 * ldx;
    xi += q0 * ldx;
    const Epi epi = epi0.shifted(q0);
    const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
    const int64_t w0 = (tile * kSpmvThreads + warp * 32) * V;   // the warp's rows: w0 .. w0 + 32 V - 1
    const int64_t mword = (tile * kSpmvThreads * V) >> 10;      // a block's rows lie in one mask word (V | 4)
    const int shift = (int)(w0 >> 5) & 31;
    const int64_t r0 = w0 + lane;
    float accr[K][V], acci[K][V];

    // the products of one diagonal with the tiles of `live`
    auto mac = [&](auto im_c, const int4 &q, int64_t base, uint32_t live) {
        constexpr bool IM = decltype(im_c)::value;
        const bool full = w0 >= q.y && w0 + 32 * V <= q.z;
        const float *pa = are + base + r0, *pb = aim + base + r0;
        const int64_t c = r0 + q.x;
        float a[V], b[V];
        bool ok[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            ok[v] = ((live >> v) & 1u) && (full || (r0 + 32 * v >= q.y && r0 + 32 * v < q.z));
            a[v] = ok[v] ? __ldcs(pa + 32 * v) : 0.f;
            if constexpr (IM) b[v] = ok[v] ? __ldcs(pb + 32 * v) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (k >= kq) break;
            const float *px = xr + k * ldx + c, *py = xi + k * ldx + c;
            float x[V], y[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                x[v] = ok[v] ? __ldg(px + 32 * v) : 0.f;
                y[v] = ok[v] ? __ldg(py + 32 * v) : 0.f;
            }
#pragma unroll
            for (int v = 0; v < V; ++v) {
                accr[k][v] = fma(a[v], x[v], accr[k][v]);
                if constexpr (IM) accr[k][v] = fma(-b[v], y[v], accr[k][v]);
                acci[k][v] = fma(a[v], y[v], acci[k][v]);
                if constexpr (IM) acci[k][v] = fma(b[v], x[v], acci[k][v]);
            }
        }
    };

    for (int pass = 0;; ++pass) {  // a second pass, with both planes, for rows that are not finite
#pragma unroll
        for (int q = 0; q < K; ++q)
#pragma unroll
            for (int v = 0; v < V; ++v) accr[q][v] = acci[q][v] = 0.f;
        for (int c0 = 0; c0 < nd; c0 += kMetaChunk) {
            const int cn = min(kMetaChunk, nd - c0);
            if (pass == 0 || nd > kMetaChunk) {
                __syncthreads();
                for (int i = threadIdx.x; i < cn; i += kSpmvThreads) {
                    const DiagMeta m = meta[c0 + i];
                    const int64_t w = (int64_t)(c0 + i) * mw + mword;
                    const uint32_t wr = tmask ? tmask[nd * mw + w] : 0xffffffffu;
                    const uint32_t wi = tmask ? tmask[2 * nd * mw + w] : 0xffffffffu;
                    sq[i] = make_int4(m.off, (int)m.lo, (int)m.hi, (int)wr);
                    sb[i] = BaseIm{m.base, wi, 0u};
                }
                __syncthreads();
            }
            if (w0 >= rows) continue;
            for (int k = 0; k < cn; ++k) {
                const int4 q = sq[k];
                const BaseIm b = sb[k];
                const uint32_t im = (b.im >> shift) & ((1u << V) - 1u);
                const uint32_t live = (((uint32_t)q.w >> shift) & ((1u << V) - 1u)) | im;
                if (w0 + 32 * V <= q.y || w0 >= q.z || !live) continue;
                if (im || pass)
                    mac(std::true_type{}, q, b.base, live);
                else
                    mac(std::false_type{}, q, b.base, live);
            }
        }
        if (pass || !tmask) break;
        uint32_t big = 0u, small = ~0u;
#pragma unroll
        for (int q = 0; q < K; ++q)
#pragma unroll
            for (int v = 0; v < V; ++v) {
                big = max(big, max(abs_hi(accr[q][v]), abs_hi(acci[q][v])));
                small = min(small, min(abs_hi(accr[q][v]), abs_hi(acci[q][v])));
            }
        const bool again = unsettled<float>(big, small);
        if (!(nd > kMetaChunk ? __syncthreads_or(again) : __any_sync(0xffffffffu, again))) break;
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
        float sr[K][1], si[K][1];
#pragma unroll
        for (int q = 0; q < K; ++q) {
            sr[q][0] = accr[q][v];
            si[q][0] = acci[q][v];
        }
        if (r0 + 32 * v < rows) epi.template apply<float, K, 1>(r0 + 32 * v, rows, kq, sr, si);
    }
}

// One row per thread in blocks of NT threads, for matrices of few rows.  With only a few warps per SM
// nothing hides the chain of one diagonal after the other, so each warp finds the diagonals that hold
// a nonzero in its 32 rows 32 at a time (one per lane, ballots for the two planes) and issues the loads
// of U of them before the multiply-adds of the first; small blocks spread the rows over more SMs.  The
// sums are those of dia_spmv_kernel, in its order.
//
// 12-qubit chain, 25 diagonals, one state: c128 6.4 us against 10.3 for dia_spmv_kernel with one row
// per thread (16.4 with two), c64 6.3 against 10.3.  The line to dia_spmv_kernel (rows x state chunks):
// float64 is bound by FP64 issue sooner and loses from there on (131,072 rows: 16.6 against 14.5 us on
// the XXZ chain, 43.8 against 38.7 on a Pauli sum; 32,768 rows: 8.3 against 10.4); float32, against 4
// rows per thread, holds to twice that (250,007 rows, 37 random diagonals: 18.6 against 21.5 us).
template <typename T>
constexpr int64_t kRowKernelMax = sizeof(T) == 8 ? 65536 : 262144;

template <typename T, int K, int NT, int U, class Epi>
__global__ void __launch_bounds__(NT)
    dia_spmv_row_kernel(const DiagMeta *__restrict__ meta, int nd, const T *__restrict__ are,
                        const T *__restrict__ aim, int rows, const T *xr, const T *xi,
                        int64_t ldx, int nrhs, int nchunk, const uint32_t *__restrict__ tmask, int64_t mw, Epi epi0) {
    __shared__ int4 sq[kMetaChunk];
    __shared__ BaseIm sb[kMetaChunk];
    const int chunk = (int)(blockIdx.x % (unsigned)nchunk);
    const int tile = blockIdx.x / (unsigned)nchunk;
    const int q0 = chunk * K;
    const int kq = min(K, nrhs - q0);
    xr += q0 * ldx;
    xi += q0 * ldx;
    const Epi epi = epi0.shifted(q0);
    const int lane = (int)threadIdx.x & 31;
    const int r = tile * NT + (int)threadIdx.x, w0 = r - lane;
    const int64_t mword = ((int64_t)tile * NT) >> 10;
    const uint32_t mine = 1u << ((r >> 5) & 31);
    T accr[K][1], acci[K][1];
    xr += r;
    xi += r;
    are += r;
    aim += r;
    if (Epi::kChained && nd == 0) dependency_wait();
    for (int pass = 0;; ++pass) {
#pragma unroll
        for (int k = 0; k < K; ++k) accr[k][0] = acci[k][0] = (T)0;
        for (int c0 = 0; c0 < nd; c0 += kMetaChunk) {
            const int cn = min(kMetaChunk, nd - c0);
            if (pass == 0 || nd > kMetaChunk) {
                __syncthreads();
                for (int i = threadIdx.x; i < cn; i += NT) {
                    const DiagMeta m = meta[c0 + i];
                    const int64_t w = (int64_t)(c0 + i) * mw + mword;
                    const uint32_t wr = tmask ? tmask[nd * mw + w] : 0xffffffffu;
                    const uint32_t wi = tmask ? tmask[2 * nd * mw + w] : 0xffffffffu;
                    sq[i] = make_int4(m.off, (int)m.lo, (int)m.hi, (int)wr);
                    sb[i] = BaseIm{m.base, wi, 0u};
                }
                __syncthreads();
                if constexpr (Epi::kChained) dependency_wait();
            }
            for (int i0 = 0; i0 < cn; i0 += 32) {
                bool re = false, im = false;
                if (i0 + lane < cn) {
                    const int4 q = sq[i0 + lane];
                    if (w0 < q.z && w0 + 32 > q.y) {
                        re = ((uint32_t)q.w & mine) != 0u;
                        im = (sb[i0 + lane].im & mine) != 0u;
                    }
                }
                uint32_t mr = __ballot_sync(0xffffffffu, re), mi = __ballot_sync(0xffffffffu, im), live = mr | mi;
                if (pass) mr = mi = live;
                struct D {
                    T x[K], y[K];
                };
                auto load = [&](int j, bool &ok, int64_t &base, D &d) {
                    const int4 q = sq[i0 + j];
                    base = sb[i0 + j].base;
                    ok = r >= q.y && r < q.z;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        if (k >= kq) break;
                        d.x[k] = ok ? load_state<Epi::kChained>(xr + k * ldx + q.x) : (T)0;
                        d.y[k] = ok ? load_state<Epi::kChained>(xi + k * ldx + q.x) : (T)0;
                    }
                };
                auto mac_re = [&](T a, const D &d) {
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        if (k >= kq) break;
                        accr[k][0] = fma(a, d.x[k], accr[k][0]);
                        acci[k][0] = fma(a, d.y[k], acci[k][0]);
                    }
                };
                auto mac_im = [&](T b, const D &d) {
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        if (k >= kq) break;
                        accr[k][0] = fma(-b, d.y[k], accr[k][0]);
                        acci[k][0] = fma(b, d.x[k], acci[k][0]);
                    }
                };
                if (!mi || !mr) {  // one plane in all of these diagonals
                    const T *pl = mi ? aim : are;
                    while (live) {
                        D d[U];
                        T a[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            if (!live) {
                                a[u] = (T)0;
                                for (int k = 0; k < K; ++k) d[u].x[k] = d[u].y[k] = (T)0;
                                continue;
                            }
                            const int j = __ffs(live) - 1;
                            live &= live - 1u;
                            bool ok;
                            int64_t base;
                            load(j, ok, base, d[u]);
                            a[u] = ok ? __ldcs(pl + base) : (T)0;
                        }
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            if (mi) mac_im(a[u], d[u]);
                            else mac_re(a[u], d[u]);
                    }
                } else {
                    while (live) {
                        D d[U];
                        T a[U], b[U];
                        uint32_t bit[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            bit[u] = live & (0u - live);
                            if (!live) continue;
                            const int j = __ffs(live) - 1;
                            live &= live - 1u;
                            bool ok;
                            int64_t base;
                            load(j, ok, base, d[u]);
                            a[u] = ok && (mr & bit[u]) ? __ldcs(are + base) : (T)0;
                            b[u] = ok && (mi & bit[u]) ? __ldcs(aim + base) : (T)0;
                        }
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            if (!(mi & bit[u])) {
                                if (bit[u]) mac_re(a[u], d[u]);
                            } else if (!(mr & bit[u])) {
                                mac_im(b[u], d[u]);
                            } else {
#pragma unroll
                                for (int k = 0; k < K; ++k) {
                                    if (k >= kq) break;
                                    accr[k][0] = fma(a[u], d[u].x[k], accr[k][0]);
                                    accr[k][0] = fma(-b[u], d[u].y[k], accr[k][0]);
                                    acci[k][0] = fma(a[u], d[u].y[k], acci[k][0]);
                                    acci[k][0] = fma(b[u], d[u].x[k], acci[k][0]);
                                }
                            }
                        }
                    }
                }
            }
        }
        if (pass || !tmask) break;
        uint32_t big = 0u, small = ~0u;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            big = max(big, max(abs_hi(accr[k][0]), abs_hi(acci[k][0])));
            small = min(small, min(abs_hi(accr[k][0]), abs_hi(acci[k][0])));
        }
        const bool again = unsettled<T>(big, small);
        if (!(nd > kMetaChunk ? __syncthreads_or(again) : __any_sync(0xffffffffu, again))) break;
    }
    if constexpr (Epi::kChained) dependents_go();
    if (r < rows) epi.template apply<T, K, 1>(r, rows, kq, accr, acci);
}

// One row per lane, the diagonals dealt out to the four warps of a block (warp w takes slots w, w + 4,
// ...), for the smallest matrices: there one warp per scheduler works through its rows' diagonals alone,
// an instruction every ten cycles or so.  The warps' partial sums are added in a fixed order, so the rounding
// differs from the other kernels' in the last bit; epilogues whose results are compared bit by bit across
// kernels keep to those (Epi::kSplit).  Metadata and masks are read by the lanes, a diagonal each, before
// dependency_wait.
//
// Against dia_spmv_row_kernel: 12-qubit Pauli sum (60 diagonals), c128, 9.2 us against 13.3; 120 terms of
// the evolution under a 13-qubit one 972 against 1,348, under the 12-qubit Ising chain 580 against 612.  The
// line (rows x state chunks): float64 is bound by FP64 issue from there on (14-qubit XXZ chain, 120
// terms: 753 against 624), float32 gains further (5 states of a 13-qubit Pauli sum: 8.7 against 14.4).
// The line goes by the call's rows and states alone, so the bits of a result do too.
template <typename T>
constexpr int64_t kSplitKernelMax = sizeof(T) == 8 ? 8192 : 32768;
template <typename T>
inline bool split_kernel_fits(int64_t rows, int nchunk) {
    return rows * nchunk <= kSplitKernelMax<T>;
}

template <typename T, int K, int U, class Epi>
__global__ void __launch_bounds__(128)
    dia_spmv_split_kernel(const DiagMeta *__restrict__ meta, int nd, const T *__restrict__ are,
                          const T *__restrict__ aim, int rows, const T *xr, const T *xi, int64_t ldx, int nrhs,
                          int nchunk, const uint32_t *__restrict__ tmask, int64_t mw, Epi epi0) {
    __shared__ T part[3][2 * K][32];
    const int chunk = (int)(blockIdx.x % (unsigned)nchunk), tile = blockIdx.x / (unsigned)nchunk;
    const int q0 = chunk * K, kq = min(K, nrhs - q0);
    const Epi epi = epi0.shifted(q0);
    const int lane = (int)threadIdx.x & 31, w = (int)threadIdx.x >> 5;
    const int r = tile * 32 + lane, w0 = tile * 32;
    xr += q0 * ldx + r;
    xi += q0 * ldx + r;
    are += r;
    aim += r;
    T accr[K][1], acci[K][1];
    for (int pass = 0;; ++pass) {   // a second pass, with both planes, for rows that are not finite
#pragma unroll
        for (int k = 0; k < K; ++k) accr[k][0] = acci[k][0] = (T)0;
        for (int c0 = w; c0 < nd; c0 += 128) {
            const int d = c0 + 4 * lane;
            int off = 0, lo = 0, hi = 0;
            int64_t base = 0;
            bool re = false, im = false;
            if (d < nd) {
                const DiagMeta m = meta[d];
                off = m.off;
                lo = (int)m.lo;
                hi = (int)m.hi;
                base = m.base;
                const int64_t at = (int64_t)d * mw + (w0 >> 10);
                const uint32_t wr = tmask ? tmask[nd * mw + at] : 0xffffffffu, wi = tmask ? tmask[2 * nd * mw + at] : 0xffffffffu;
                if (w0 < hi && w0 + 32 > lo) {
                    re = (wr >> ((w0 >> 5) & 31)) & 1u;
                    im = (wi >> ((w0 >> 5) & 31)) & 1u;
                }
            }
            uint32_t mr = __ballot_sync(0xffffffffu, re), mi = __ballot_sync(0xffffffffu, im), live = mr | mi;
            if (pass) mr = mi = live;
            if constexpr (Epi::kChained) dependency_wait();
            while (live) {
                T a[U], b[U], x[U][K], y[U][K];
                uint32_t bit[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    bit[u] = live & (0u - live);
                    if (!live) continue;
                    const int j = __ffs(live) - 1;
                    live &= live - 1u;
                    const int o = __shfl_sync(0xffffffffu, off, j), l = __shfl_sync(0xffffffffu, lo, j),
                              h = __shfl_sync(0xffffffffu, hi, j);
                    const int64_t vb = __shfl_sync(0xffffffffu, base, j);
                    const bool ok = r >= l && r < h;
                    a[u] = ok && (mr & bit[u]) ? __ldcs(are + vb) : (T)0;
                    b[u] = ok && (mi & bit[u]) ? __ldcs(aim + vb) : (T)0;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        if (k >= kq) break;
                        x[u][k] = ok ? load_state<Epi::kChained>(xr + k * ldx + o) : (T)0;
                        y[u][k] = ok ? load_state<Epi::kChained>(xi + k * ldx + o) : (T)0;
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (mr & bit[u])
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            if (k >= kq) break;
                            accr[k][0] = fma(a[u], x[u][k], accr[k][0]);
                            acci[k][0] = fma(a[u], y[u][k], acci[k][0]);
                        }
                    if (mi & bit[u])
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            if (k >= kq) break;
                            accr[k][0] = fma(-b[u], y[u][k], accr[k][0]);
                            acci[k][0] = fma(b[u], x[u][k], acci[k][0]);
                        }
                }
            }
        }
        if constexpr (Epi::kChained) dependency_wait();   // (a warp without diagonals has not waited yet)
        if (w > 0)
#pragma unroll
            for (int k = 0; k < K; ++k) {
                part[w - 1][2 * k][lane] = accr[k][0];
                part[w - 1][2 * k + 1][lane] = acci[k][0];
            }
        __syncthreads();
        bool again = false;
        if (w == 0) {
            uint32_t big = 0u, small = ~0u;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                accr[k][0] = (accr[k][0] + part[0][2 * k][lane]) + (part[1][2 * k][lane] + part[2][2 * k][lane]);
                acci[k][0] = (acci[k][0] + part[0][2 * k + 1][lane]) + (part[1][2 * k + 1][lane] + part[2][2 * k + 1][lane]);
                big = max(big, max(abs_hi(accr[k][0]), abs_hi(acci[k][0])));
                small = min(small, min(abs_hi(accr[k][0]), abs_hi(acci[k][0])));
            }
            again = unsettled<T>(big, small);
        }
        if (pass || !tmask || !__syncthreads_or(again)) break;
    }
    if constexpr (Epi::kChained) dependents_go();
    if (w == 0 && r < rows) epi.template apply<T, K, 1>(r, rows, kq, accr, acci);
}

// ---- float variant with L2 prefetch of the matrix and shuffled state windows ----------------------
//
// The register kernel above waits, on every diagonal, for the HBM latency of its matrix vector:
// a warp has one diagonal's loads in flight, and a few dozen warps per SM do not cover the
// latency (profiles: ~30 % of HBM bandwidth, long-scoreboard stalls).  Here lane 0 of each warp
// asks L2 for the warp's 128-row strip of the matrix PF diagonals ahead with one bulk prefetch
// per array (cp.async.bulk.prefetch.L2: no registers, no shared memory), so the loads the warp
// then issues hit L2.
//
// The state windows of a diagonal whose offset is not a multiple of 4 start between 16-byte
// vectors.  The offset is the same for the whole warp, so each lane loads its aligned vector
// and takes the next one from the neighbouring lane (lane 31 loads it): one 16-byte load per
// lane instead of four 4-byte loads.  Strips that a diagonal covers only in part (at the
// matrix's edges) take the element-wise path of the register kernel.
//
// Needs cols % 4 == 0, ldx % 4 == 0 and 16-byte aligned x arrays (checked by the launcher);
// then every x read stays below column cols.

// Ask L2 for [p, p + bytes): p 16-byte aligned, bytes a multiple of 16.  The lines come in with
// evict-first priority, like the streaming loads that will read them, so that they do not push
// the re-read state windows out of L2.
__device__ __forceinline__ void prefetch_l2_bulk(const void *p, unsigned bytes) {
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(policy));
    asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;\n" ::"l"(p), "r"(bytes), "l"(policy)
                 : "memory");
}

// Rows [w0, w0 + 128) of diagonal m, clipped to the diagonal's rows rounded out to 32 values
// (inside the allocation: the first diagonal starts 32 values in and 32 values follow the last;
// base is a multiple of 32, so the clipped range starts on a 128-byte boundary).
__device__ __forceinline__ void prefetch_strip(const DiagMeta &m, int64_t w0, const float *are,
                                               const float *aim) {
    const int64_t a = w0 > (m.lo & ~int64_t(31)) ? w0 : (m.lo & ~int64_t(31));
    const int64_t hi32 = (m.hi + 31) & ~int64_t(31);
    const int64_t b = (w0 + 128) < hi32 ? (w0 + 128) : hi32;
    if (a >= b) return;
    prefetch_l2_bulk(are + m.base + a, (unsigned)(b - a) * 4u);
    prefetch_l2_bulk(aim + m.base + a, (unsigned)(b - a) * 4u);
}

// The four values x[c .. c+3] for a warp whose lanes own consecutive 4-row groups, c - s the
// lane's aligned vector (s = c & 3, the same in every lane).
__device__ __forceinline__ void shifted_window(float (&out)[4], const float *aligned_p, int s, int lane) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(aligned_p));
    if (s == 0) {
        out[0] = a.x;
        out[1] = a.y;
        out[2] = a.z;
        out[3] = a.w;
        return;
    }
    float n0 = __shfl_down_sync(0xffffffffu, a.x, 1);
    float n1 = __shfl_down_sync(0xffffffffu, a.y, 1);
    float n2 = __shfl_down_sync(0xffffffffu, a.z, 1);
    if (lane == 31) {
        const float4 b = __ldg(reinterpret_cast<const float4 *>(aligned_p + 4));
        n0 = b.x;
        n1 = b.y;
        n2 = b.z;
    }
    if (s == 1) {
        out[0] = a.y;
        out[1] = a.z;
        out[2] = a.w;
        out[3] = n0;
    } else if (s == 2) {
        out[0] = a.z;
        out[1] = a.w;
        out[2] = n0;
        out[3] = n1;
    } else {
        out[0] = a.w;
        out[1] = n0;
        out[2] = n1;
        out[3] = n2;
    }
}

template <int K, int PF, class Epi>
__global__ void __launch_bounds__(kSpmvThreads)
    dia_spmv_pf_kernel(const DiagMeta *__restrict__ meta, int nd, const float *__restrict__ are,
                       const float *__restrict__ aim, int64_t rows, const float *__restrict__ xr,
                       const float *__restrict__ xi, int64_t ldx, int kq, Epi epi) {
    constexpr int V = 4;
    __shared__ DiagMeta sm[kMetaChunk];
    const int lane = threadIdx.x & 31;
    const int64_t r0 = ((int64_t)blockIdx.x * kSpmvThreads + threadIdx.x) * V;
    const int64_t w0 = r0 - (int64_t)V * lane;  // first row of the warp's 128-row strip
    float accr[K][V], acci[K][V];
#pragma unroll
    for (int q = 0; q < K; ++q)
#pragma unroll
        for (int v = 0; v < V; ++v) accr[q][v] = acci[q][v] = 0.f;

    for (int c0 = 0; c0 < nd; c0 += kMetaChunk) {
        const int cn = min(kMetaChunk, nd - c0);
        __syncthreads();
        for (int i = threadIdx.x; i < cn; i += kSpmvThreads) sm[i] = meta[c0 + i];
        __syncthreads();
        if (w0 >= rows) continue;  // the whole warp is past the last row
        if (PF > 0 && lane == 0)
            for (int k = 0; k < PF && k < cn; ++k) prefetch_strip(sm[k], w0, are, aim);
        for (int k = 0; k < cn; ++k) {
            if (PF > 0 && lane == 0 && k + PF < cn) prefetch_strip(sm[k + PF], w0, are, aim);
            const int64_t lo = sm[k].lo, hi = sm[k].hi;
            if (w0 >= hi || w0 + 32 * V <= lo) continue;  // the same for the whole warp
            const int64_t base = sm[k].base;
            const int64_t c = r0 + sm[k].off;
            if (w0 >= lo && w0 + 32 * V <= hi) {
                // the strip lies inside the diagonal: every lane has 4 valid rows
                float ar[V], ai[V];
                load_vec_stream<float, V>(ar, are + base + r0);
                load_vec_stream<float, V>(ai, aim + base + r0);
                const int s = (int)(c & 3);
                const int64_t ca = c - s;
#pragma unroll
                for (int q = 0; q < K; ++q) {
                    if (q >= kq) break;
                    float xrv[V], xiv[V];
                    shifted_window(xrv, xr + q * ldx + ca, s, lane);
                    shifted_window(xiv, xi + q * ldx + ca, s, lane);
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        accr[q][v] = fmaf(ar[v], xrv[v], accr[q][v]);
                        accr[q][v] = fmaf(-ai[v], xiv[v], accr[q][v]);
                        acci[q][v] = fmaf(ar[v], xiv[v], acci[q][v]);
                        acci[q][v] = fmaf(ai[v], xrv[v], acci[q][v]);
                    }
                }
            } else {
                // edge strip: element-wise, rows outside [lo, hi) (and past the last row) masked
                if (r0 >= rows || r0 + V <= lo || r0 >= hi) continue;
                float ar[V], ai[V];
                load_vec_stream<float, V>(ar, are + base + r0);
                load_vec_stream<float, V>(ai, aim + base + r0);
#pragma unroll
                for (int v = 0; v < V; ++v)
                    if (r0 + v < lo || r0 + v >= hi) ar[v] = ai[v] = 0.f;
#pragma unroll
                for (int q = 0; q < K; ++q) {
                    if (q >= kq) break;
                    const float *pxr = xr + q * ldx + c, *pxi = xi + q * ldx + c;
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        const bool ok = (r0 + v >= lo) && (r0 + v < hi);
                        const float xv = ok ? __ldg(pxr + v) : 0.f, yv = ok ? __ldg(pxi + v) : 0.f;
                        accr[q][v] = fmaf(ar[v], xv, accr[q][v]);
                        accr[q][v] = fmaf(-ai[v], yv, accr[q][v]);
                        acci[q][v] = fmaf(ar[v], yv, acci[q][v]);
                        acci[q][v] = fmaf(ai[v], xv, acci[q][v]);
                    }
                }
            }
        }
    }
    if (r0 < rows) epi.template apply<float, K, V>(r0, rows, kq, accr, acci);
}

// Whether the prefetching kernel may run on these state arrays (see its notes).
inline bool pf_kernel_fits(const Matrix &A, const float *xr, const float *xi, int64_t ldx, int nrhs) {
    return A.cols % 4 == 0 && (nrhs == 1 || ldx % 4 == 0) && (reinterpret_cast<uintptr_t>(xr) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(xi) & 15) == 0;
}

// Store y = A x.  (kChained: whether kernels with this epilogue are launched with launch_chained; kSplit:
// whether dia_spmv_split_kernel may run them.)
template <typename T>
struct EpiStore {
    static constexpr bool kChained = false, kSplit = true;
    T *yr, *yi;
    int64_t ldy;
    template <typename U, int K, int V>
    __device__ __forceinline__ void apply(int64_t r0, int64_t rows, int kq, U (&ar)[K][V], U (&ai)[K][V]) const {
#pragma unroll
        for (int q = 0; q < K; ++q) {
            if (q >= kq) break;
            T *pr = yr + q * ldy + r0, *pi = yi + q * ldy + r0;
            if (V > 1 && r0 + V <= rows && aligned_to<V * sizeof(T)>(pr) && aligned_to<V * sizeof(T)>(pi)) {
                using VT = typename Vec<T, V>::type;
                VT a, b;
                if constexpr (V == 2) {
                    a = VT{ar[q][0], ar[q][1]};
                    b = VT{ai[q][0], ai[q][1]};
                } else if constexpr (V == 4) {
                    a = VT{ar[q][0], ar[q][1], ar[q][2], ar[q][3]};
                    b = VT{ai[q][0], ai[q][1], ai[q][2], ai[q][3]};
                }
                if constexpr (V > 1) {
                    *reinterpret_cast<VT *>(pr) = a;
                    *reinterpret_cast<VT *>(pi) = b;
                }
            } else {
#pragma unroll
                for (int v = 0; v < V; ++v)
                    if (r0 + v < rows) {
                        pr[v] = ar[q][v];
                        pi[v] = ai[q][v];
                    }
            }
        }
    }
};

// One Taylor term of the reference's time evolution (src/spHamSim_gpu_all_fused.cu:206-229):
// term = (-i * scale) * (A term_in), i.e. (re, im) = (s_im * scale, -s_re * scale); acc += term.
// With init set, acc = init + term instead (the first term of a step starts the sum from the
// state itself, saving the copy).  Vectors and accumulator of type T.
template <typename T>
struct EpiTaylor {
    static constexpr bool kChained = true, kSplit = true;
    T *tr, *ti;      // term out
    T *accr, *acci;  // running sum
    const T *initr, *initi;
    int64_t ld;
    T scale;
    template <typename U, int K, int V>
    __device__ __forceinline__ void apply(int64_t r0, int64_t rows, int kq, U (&sr)[K][V], U (&si)[K][V]) const {
#pragma unroll
        for (int q = 0; q < K; ++q)
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const int64_t r = r0 + v;
                if (q < kq && r < rows) {
                    const int64_t i = q * ld + r;
                    const T a = sr[q][v], b = si[q][v];
                    const T nr = b * scale, ni = -a * scale;
                    tr[i] = nr;
                    ti[i] = ni;
                    if (initr) {
                        accr[i] = initr[i] + nr;
                        acci[i] = initi[i] + ni;
                    } else {
                        accr[i] += nr;
                        acci[i] += ni;
                    }
                }
            }
    }
};

inline unsigned spmv_blocks(int64_t rows, int V) {
    const int64_t per = (int64_t)kSpmvThreads * V;
    return (unsigned)((rows + per - 1) / per);
}

// Launch shape of the SpMV family: at most kmax states per launch (the matrix is read once per
// launch), vr rows per thread (the tile of a block is 256 * vr rows).  vr = 0 picks the widest
// 16-byte vector.
struct SpmvCfg {
    int kmax = 8;
    int vr = 0;
    int pipe = 0;  // kernel variant: 0 registers; float kernels with 4 rows per thread: 1 cp.async pipeline,
                   // shuffled windows with L2 prefetch 4 (2) or 8 (3) diagonals ahead or none (4)
};

template <typename T, int K, class Epi, int VR, int... More>
void launch_vr(int vr, const Matrix &A, const T *xr, const T *xi, int64_t ldx, int nrhs, int nchunk,
               const Epi &e, cudaStream_t s, const uint32_t *tmask, bool chained) {
    if constexpr (sizeof...(More) > 0) {
        if (vr != VR) {
            launch_vr<T, K, Epi, More...>(vr, A, xr, xi, ldx, nrhs, nchunk, e, s, tmask, chained);
            return;
        }
    }
    if constexpr (VR == 1 && K <= 2) {
        constexpr int NT = 64, U = K == 1 ? 4 : 2;
        const int64_t blocks = (A.rows + NT - 1) / NT * nchunk;
        if constexpr (Epi::kSplit) {
            if (split_kernel_fits<T>(A.rows, nchunk)) {
                launch_chained(chained, dia_spmv_split_kernel<T, K, U, Epi>, (unsigned)((A.rows + 31) / 32 * nchunk), 128, s,
                               A.d_meta, A.nd, (const T *)A.re, (const T *)A.im, (int)A.rows, xr, xi, ldx, nrhs, nchunk,
                               tmask, tile_mask_words(A.rows), e);
                return;
            }
        }
        if (A.rows * nchunk <= kRowKernelMax<T>) {
            launch_chained(chained, dia_spmv_row_kernel<T, K, NT, U, Epi>, (unsigned)blocks, NT, s, A.d_meta, A.nd,
                           (const T *)A.re, (const T *)A.im, (int)A.rows, xr, xi, ldx, nrhs, nchunk, tmask,
                           tile_mask_words(A.rows), e);
            return;
        }
    }
    launch_chained(chained, dia_spmv_kernel<T, K, VR, Epi>, spmv_blocks(A.rows, VR) * (unsigned)nchunk, kSpmvThreads, s,
                   A.d_meta, A.nd, (const T *)A.re, (const T *)A.im, A.rows, xr, xi, ldx, nrhs, nchunk, tmask,
                   tile_mask_words(A.rows), e);
}

// One launch over all right-hand sides, in chunks of up to cfg.kmax (<= 8) states per block
// (the kernel instantiated for 1, 2, 4 or 8 states, unused slots of the last chunk masked); the
// chunks of a row tile run side by side (see dia_spmv_kernel).  VRs lists the rows-per-thread
// variants compiled for this epilogue (the first is the default).  Epi must offer
// `shifted(q0)` on host and device, the same epilogue for right-hand sides q0.. .  tmask: A's
// zero-tile mask (build_tile_mask), or NULL to visit every tile.  chained: see launch_chained.
template <typename T, class Epi, int... VRs>
int launch_dia_spmv_rhs_cfg(const Matrix &A, const T *xr, const T *xi, int64_t ldx, int nrhs, Epi epi,
                            cudaStream_t s, SpmvCfg cfg, const uint32_t *tmask = nullptr, bool chained = false) {
    if (A.rows == 0 || nrhs <= 0) return DIAQ_OK;
    int k = cfg.kmax >= 8 ? 8 : cfg.kmax >= 4 ? 4 : cfg.kmax >= 2 ? 2 : 1;
    while (k > 1 && k / 2 >= nrhs) k /= 2;  // no wider than the states need
    const int vr = cfg.vr > 0 ? cfg.vr : VecOf<T>::V;
    const int nchunk = (nrhs + k - 1) / k;
    if ((uint64_t)spmv_blocks(A.rows, vr) * (uint64_t)nchunk > 0x7fffffffull)
        return set_error(DIAQ_ERR_UNSUPPORTED, "spmv: too many row tiles x state chunks for one launch");
    if (k == 8)
        launch_vr<T, 8, Epi, VRs...>(vr, A, xr, xi, ldx, nrhs, nchunk, epi, s, tmask, chained);
    else if (k == 4)
        launch_vr<T, 4, Epi, VRs...>(vr, A, xr, xi, ldx, nrhs, nchunk, epi, s, tmask, chained);
    else if (k == 2)
        launch_vr<T, 2, Epi, VRs...>(vr, A, xr, xi, ldx, nrhs, nchunk, epi, s, tmask, chained);
    else
        launch_vr<T, 1, Epi, VRs...>(vr, A, xr, xi, ldx, nrhs, nchunk, epi, s, tmask, chained);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

// The shuffled-window float kernel over the states in chunks of up to kmax; variant 2 / 3
// prefetches the matrix 4 / 8 diagonals ahead, variant 4 does not prefetch.  Falls back to the
// register kernel (4 rows per thread) where pf_kernel_fits does not hold.
template <int K, class Epi>
void launch_pf_k(int variant, const Matrix &A, const float *xr, const float *xi, int64_t ldx, int kq, const Epi &e,
                 cudaStream_t s) {
    const unsigned g = spmv_blocks(A.rows, 4);
    const float *are = (const float *)A.re, *aim = (const float *)A.im;
    if (variant == 3)
        dia_spmv_pf_kernel<K, 8, Epi><<<g, kSpmvThreads, 0, s>>>(A.d_meta, A.nd, are, aim, A.rows, xr, xi, ldx, kq, e);
    else if (variant == 4)
        dia_spmv_pf_kernel<K, 0, Epi><<<g, kSpmvThreads, 0, s>>>(A.d_meta, A.nd, are, aim, A.rows, xr, xi, ldx, kq, e);
    else
        dia_spmv_pf_kernel<K, 4, Epi><<<g, kSpmvThreads, 0, s>>>(A.d_meta, A.nd, are, aim, A.rows, xr, xi, ldx, kq, e);
}

template <class Epi>
int launch_dia_spmv_pf(const Matrix &A, const float *xr, const float *xi, int64_t ldx, int nrhs, Epi epi,
                       cudaStream_t s, int kmax, int variant, int *launches) {
    if (A.rows == 0 || nrhs <= 0) return DIAQ_OK;
    if (!pf_kernel_fits(A, xr, xi, ldx, nrhs)) {
        ++*launches;
        return launch_dia_spmv_rhs_cfg<float, Epi, 4>(A, xr, xi, ldx, nrhs, epi, s, SpmvCfg{kmax, 4, 0});
    }
    kmax = kmax >= 8 ? 8 : kmax >= 4 ? 4 : kmax >= 2 ? 2 : 1;
    int q0 = 0;
    while (q0 < nrhs) {
        const int left = nrhs - q0;
        const int kq = left < kmax ? left : kmax;
        const float *pxr = xr + q0 * ldx, *pxi = xi + q0 * ldx;
        const Epi e = epi.shifted(q0);
        if (kq > 4)
            launch_pf_k<8, Epi>(variant, A, pxr, pxi, ldx, kq, e, s);
        else if (kq > 2)
            launch_pf_k<4, Epi>(variant, A, pxr, pxi, ldx, kq, e, s);
        else if (kq == 2)
            launch_pf_k<2, Epi>(variant, A, pxr, pxi, ldx, kq, e, s);
        else
            launch_pf_k<1, Epi>(variant, A, pxr, pxi, ldx, kq, e, s);
        q0 += kq;
        ++*launches;
    }
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

// The default shape.  One row per thread for float64 (bound by FP64 issue or by latency: 76 us against
// 83 with two rows on the 20-qubit chain, 43 against 53 on a 250,007-row band, where unaligned windows
// fall apart into single loads) and for few rows (the row kernel); 16-byte vectors of 4 rows for float32
// above that (35 us against 62 on the 20-qubit chain).
//
// Two states per block rather than eight: 38 against 79 us for 11 float32 states of 65,536 rows, 40
// against 46 for 5 of 250,007 (before dia_spmv_strip_kernel took the latter).  Where the matrix no longer
// fits in L2 beside the chunks it holds as well: 1,000,001 rows of 41 complex diagonals, 8 / 32 states,
// 173 / 817 us in float32 (eight states per block, before the choice of planes: 273 / 1,150), float64
// 1,098 / 4,347 (1,158 / 4,543); 20-qubit chain, 16 states, float32 277 (358).
//
// One state per block for an odd number of them in float64, where the last block's empty slot takes as
// long as a state: 150,001-row band, 20 / 45 diagonals, 3 states 39 / 80 us against 51 / 102; 16-qubit
// chain, 5 states 25.6 against 28.8.  Not where that takes the call past the line of a kernel for fewer
// rows (12-qubit Pauli sum, 3 states, 10.9 against 8.4; 5 states of 20,001 rows 26.9 against 25.3) -- but
// for 3 states at the second line (15-qubit Ising chain 12.9 against 16.9).
template <typename T>
SpmvCfg default_cfg(int64_t rows, int nrhs) {
    int k = nrhs == 1 ? 1 : 2;
    if (sizeof(T) == 8 && nrhs % 2) {
        auto kernel = [&](int groups) {
            return split_kernel_fits<T>(rows, groups) ? 0 : rows * groups <= kRowKernelMax<T> ? 1 : 2;
        };
        const int pairs = kernel((nrhs + 1) / 2);
        if (pairs == kernel(nrhs) || (nrhs == 3 && pairs == 1)) k = 1;
    }
    const bool few = rows * ((nrhs + k - 1) / k) <= kRowKernelMax<T>;
    return SpmvCfg{k, sizeof(T) == 8 || few ? 1 : 4, 0};
}

// Whether dia_spmv_strip_kernel takes a product whose default is the kernel of two states and four rows:
// it needs fewer passes over the matrix (3 states, or 5 and more); the two-state shape's blocks are more
// than run at a time (four per SM), so that its last wave is mostly empty (33 diagonals: 200,001
// rows, 5 states, 587 blocks 26 us against 29; 220,001 rows, 645 blocks, 34 against 27); and at least
// half of the windows are not on 16-byte boundaries (18-qubit chain, 8 states: 41 us against 45).
inline bool strips_pay(const Matrix &A, const float *xr, const float *xi, int64_t ldx, int nrhs) {
    if ((nrhs + 2) / 3 >= (nrhs + 1) / 2) return false;
    if (A.rows > 0x7fffffffll * 1024 / nrhs) return false;
    if ((int64_t)spmv_blocks(A.rows, kStripRows) * ((nrhs + 1) / 2) <= 4 * (int64_t)num_sms()) return false;
    if (ldx % 4 || ((reinterpret_cast<uintptr_t>(xr) | reinterpret_cast<uintptr_t>(xi)) & 15u)) return true;
    int32_t odd = 0;
    for (int32_t d : A.off) odd += (d & 3) != 0;
    return 2 * (int64_t)odd >= A.nd;
}

template <class Epi>
int launch_dia_spmv_strips(const Matrix &A, const float *xr, const float *xi, int64_t ldx, int nrhs, Epi epi,
                           cudaStream_t s, const uint32_t *tmask) {
    const int nchunk = (nrhs + kStripStates - 1) / kStripStates;
    dia_spmv_strip_kernel<kStripStates, kStripRows, Epi>
        <<<spmv_blocks(A.rows, kStripRows) * (unsigned)nchunk, kSpmvThreads, 0, s>>>(
            A.d_meta, A.nd, (const float *)A.re, (const float *)A.im, A.rows, xr, xi, ldx, nrhs, nchunk, tmask,
            tile_mask_words(A.rows), epi);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

template <typename T, class Epi>
int launch_dia_spmv_rhs(const Matrix &A, const T *xr, const T *xi, int64_t ldx, int nrhs, Epi epi,
                        cudaStream_t s, const uint32_t *tmask, bool chained = false) {
    const SpmvCfg cfg = default_cfg<T>(A.rows, nrhs);
    if constexpr (sizeof(T) == 4 && !Epi::kChained)
        if (cfg.vr == kStripRows && strips_pay(A, xr, xi, ldx, nrhs))
            return launch_dia_spmv_strips(A, xr, xi, ldx, nrhs, epi, s, tmask);
    if constexpr (sizeof(T) == 4)
        return launch_dia_spmv_rhs_cfg<T, Epi, 4, 1>(A, xr, xi, ldx, nrhs, epi, s, cfg, tmask, chained);
    else
        return launch_dia_spmv_rhs_cfg<T, Epi, 1>(A, xr, xi, ldx, nrhs, epi, s, cfg, tmask, chained);
}

template <typename T>
struct EpiStoreRhs : EpiStore<T> {
    __host__ __device__ EpiStoreRhs shifted(int q0) const {
        EpiStoreRhs e = *this;
        e.yr += q0 * this->ldy;
        e.yi += q0 * this->ldy;
        return e;
    }
};

template <typename T>
struct EpiTaylorRhs : EpiTaylor<T> {
    __host__ __device__ EpiTaylorRhs shifted(int q0) const {
        EpiTaylorRhs e = *this;
        const int64_t o = q0 * this->ld;
        e.tr += o;
        e.ti += o;
        e.accr += o;
        e.acci += o;
        if (e.initr) {
            e.initr += o;
            e.initi += o;
        }
        return e;
    }
};

}  // namespace diaq_gb300
