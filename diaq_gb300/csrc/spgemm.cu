// Diagonal-pair SpGEMM C = A B with its structural dry-run on the device.
// Replaces product / product_device / product_cuda (src/spGEMM.cpp:303-538,
// src/spGEMM_gpu.cu:25-161).
//
// Dry-run: every pair (dA, dB) marks dC = dA + dB in a flag array over the whole offset range
// [-(rowsA-1), colsB-1]; an exclusive prefix sum over the flags numbers the marked offsets, so
// compaction yields them ascending and distinct -- a counting sort, exact by construction, the
// set the reference collects in a std::map (src/spGEMM.cpp:346-369).
//
// Numeric pass: in row-indexed form C[r, dC] = sum_a A[r, dA_a] * B[r + dA_a, dC - dA_a].  The (A, B)
// slot pairs of every C diagonal are listed once on the device; a warp owns a strip of rows, walks the
// pairs of a run of C diagonals and accumulates the shifted products -- the SpMV access pattern with
// B's diagonal in place of x.  Pairs of one C diagonal are summed in A-slot order, as
// src/spGEMM_gpu.cu:55-77 and src/spGEMM.cpp:425-493 do.
#include <algorithm>

#include "spmv_kernel.cuh"

namespace diaq_gb300 {

// ---- dry-run -----------------------------------------------------------------------------------
__global__ void mark_pairs_kernel(const DiagMeta *__restrict__ mA, int ndA, const DiagMeta *__restrict__ mB,
                                  int ndB, int64_t lo, int64_t hi, uint8_t *__restrict__ flags) {
    const int64_t n = (int64_t)ndA * ndB;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t dc = (int64_t)mA[p / ndB].off + mB[p % ndB].off;
        if (dc >= lo && dc <= hi) flags[dc - lo] = 1;  // benign race: every writer stores 1
    }
}

constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;  // flags per thread per block pass
constexpr int64_t kScanTile = (int64_t)kScanThreads * kScanItems;

// Per tile: number of set flags.
__global__ void count_tiles_kernel(const uint8_t *__restrict__ flags, int64_t n, int32_t *__restrict__ tile_count) {
    __shared__ int red[kScanThreads / 32];
    const int64_t t0 = blockIdx.x * kScanTile;
    int v = 0;
    for (int i = 0; i < kScanItems; ++i) {
        const int64_t j = t0 + (int64_t)i * kScanThreads + threadIdx.x;
        if (j < n) v += flags[j];
    }
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = threadIdx.x < kScanThreads / 32 ? red[threadIdx.x] : 0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) tile_count[blockIdx.x] = v;
    }
}

// Exclusive scan of the tile counts in one block (loops over chunks); the total goes to *total.
__global__ void scan_tiles_kernel(int32_t *__restrict__ tile_count, int64_t ntiles, int32_t *__restrict__ total) {
    __shared__ int32_t buf[1024];
    __shared__ int32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int64_t c0 = 0; c0 < ntiles; c0 += 1024) {
        const int64_t j = c0 + threadIdx.x;
        int32_t v = j < ntiles ? tile_count[j] : 0;
        buf[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < 1024; o <<= 1) {  // Hillis-Steele inclusive scan
            int32_t add = threadIdx.x >= o ? buf[threadIdx.x - o] : 0;
            __syncthreads();
            buf[threadIdx.x] += add;
            __syncthreads();
        }
        if (j < ntiles) tile_count[j] = carry + buf[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry += buf[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// Write the offsets of the set flags, ascending.
__global__ void compact_kernel(const uint8_t *__restrict__ flags, int64_t n, int64_t lo,
                               const int32_t *__restrict__ tile_base, int32_t *__restrict__ out) {
    __shared__ int32_t buf[kScanThreads];
    const int64_t t0 = blockIdx.x * kScanTile;
    int32_t base = tile_base[blockIdx.x];
    for (int i = 0; i < kScanItems; ++i) {
        const int64_t j = t0 + (int64_t)i * kScanThreads + threadIdx.x;
        const int32_t f = (j < n) ? flags[j] : 0;
        buf[threadIdx.x] = f;
        __syncthreads();
        for (int o = 1; o < kScanThreads; o <<= 1) {
            int32_t add = threadIdx.x >= o ? buf[threadIdx.x - o] : 0;
            __syncthreads();
            buf[threadIdx.x] += add;
            __syncthreads();
        }
        if (f) out[base + buf[threadIdx.x] - 1] = (int32_t)(j + lo);
        const int32_t chunk_total = buf[kScanThreads - 1];
        __syncthreads();
        base += chunk_total;
    }
}

// Symbolic phase on the device: result offsets (ascending, distinct) to the host vector.
int spgemm_symbolic(const Matrix &A, const Matrix &B, std::vector<int32_t> &offC, cudaStream_t s) {
    if (A.prec == DIAQ_C128F2) return set_error(DIAQ_ERR_UNSUPPORTED, "product: convert a c128f2 matrix to c128 first");
    offC.clear();
    if (A.cols != B.rows) return set_error(DIAQ_ERR_INVALID, "diaQMatrix product_cuda: dimension mismatch.");
    if (A.nd == 0 || B.nd == 0 || A.rows == 0 || B.cols == 0) return DIAQ_OK;
    const int64_t lo = -(A.rows - 1), hi = B.cols - 1;
    const int64_t range = hi - lo + 1;
    const int64_t ntiles = (range + kScanTile - 1) / kScanTile;
    // one scratch allocation: flags | tile counts | output (the count, then the offsets)
    const size_t fbytes = (size_t)((range + 15) / 16 * 16);
    const size_t tbytes = sizeof(int32_t) * (size_t)(ntiles + 1);
    const int64_t maxout = std::min<int64_t>((int64_t)A.nd * B.nd, range);
    const size_t obytes = sizeof(int32_t) * (size_t)(maxout + 1);
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    uint8_t *scratch = nullptr;
    DQ_CUDA(dev_malloc_async(&scratch, up(fbytes) + up(tbytes) + up(obytes), s));
    uint8_t *flags = scratch;
    int32_t *tiles = (int32_t *)(scratch + up(fbytes));
    int32_t *dout = (int32_t *)((uint8_t *)tiles + up(tbytes));
    int st = DIAQ_OK;
    cudaError_t e = cudaMemsetAsync(flags, 0, fbytes, s);
    if (e == cudaSuccess) {
        const int64_t pairs = (int64_t)A.nd * B.nd;
        const int grid = (int)std::min<int64_t>((pairs + 255) / 256, 8 * num_sms());
        mark_pairs_kernel<<<grid, 256, 0, s>>>(A.d_meta, A.nd, B.d_meta, B.nd, lo, hi, flags);
        count_tiles_kernel<<<(unsigned)ntiles, kScanThreads, 0, s>>>(flags, range, tiles);
        scan_tiles_kernel<<<1, 1024, 0, s>>>(tiles, ntiles, dout);
        compact_kernel<<<(unsigned)ntiles, kScanThreads, 0, s>>>(flags, range, lo, tiles, dout + 1);
        e = cudaGetLastError();
    }
    // the count with every offset there can be in one copy, unless those are many
    const int64_t first = maxout <= (1 << 18) ? maxout + 1 : 1;
    std::vector<int32_t> got((size_t)first, 0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(got.data(), dout, sizeof(int32_t) * (size_t)first, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && got[0] > 0) {
        if (first > 1) {
            offC.assign(got.begin() + 1, got.begin() + 1 + got[0]);
        } else {
            offC.resize((size_t)got[0]);
            e = cudaMemcpyAsync(offC.data(), dout + 1, sizeof(int32_t) * offC.size(), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        }
    }
    if (e != cudaSuccess) st = cuda_status(e, "spgemm dry-run", __FILE__, __LINE__);
    cudaFreeAsync(scratch, s);
    return st;
}

// ---- numeric pass -------------------------------------------------------------------------------
// Pair lists first: for every C diagonal c, the (A slot, B slot) pairs with dA + dB = dC whose
// rows can overlap C's, in A-slot order (the reference's summation order, src/spGEMM.cpp:346-378).
// One warp per C diagonal counts them, the host scans the counts, the same warp writes them (one thread
// per diagonal took 745 us for the 2,047 x 2,047 pairs of a full 1,024-row square, a warp 35 us).
// The numeric kernel then walks only the pairs of its C diagonal -- an earlier version scanned
// every A diagonal for every C diagonal and row tile (41 candidates for ~2.3 pairs on the
// 20-qubit XXZ H H) and spent half its instructions on that.

__device__ __forceinline__ bool pair_rows(const DiagMeta &ma, const DiagMeta &mb, const DiagMeta &mc, int64_t &lo,
                                          int64_t &hi) {
    // rows r with A valid (ma.lo <= r < ma.hi), B valid (mb.lo <= r + dA < mb.hi), C valid
    lo = max(max(ma.lo, mb.lo - (int64_t)ma.off), mc.lo);
    hi = min(min(ma.hi, mb.hi - (int64_t)ma.off), mc.hi);
    return lo < hi;
}

// One warp per C diagonal, 32 A slots at a time (a ballot keeps the slot order).  fill == nullptr: count
// the pairs of each C diagonal into cnt; else write them at start[c].
__global__ void spgemm_pairs_kernel(const DiagMeta *__restrict__ mA, int ndA, const DiagMeta *__restrict__ mB,
                                    const int32_t *__restrict__ bslot, int64_t bmin, int64_t bmax,
                                    const DiagMeta *__restrict__ mC, int ndC, int32_t *__restrict__ cnt,
                                    const int64_t *__restrict__ start, int2 *__restrict__ fill) {
    const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
    for (int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ndC; c += warps) {
        const DiagMeta mc = mC[c];
        int64_t w = fill ? start[c] : 0;
        int32_t n = 0;
        for (int a0 = 0; a0 < ndA; a0 += 32) {
            const int a = a0 + lane;
            int32_t b = -1;
            if (a < ndA) {
                const DiagMeta ma = mA[a];
                const int64_t db = (int64_t)mc.off - ma.off;
                if (db >= bmin && db <= bmax) b = bslot[db - bmin];
                int64_t lo, hi;
                if (b >= 0 && !pair_rows(ma, mB[b], mc, lo, hi)) b = -1;
            }
            const uint32_t in = __ballot_sync(0xffffffffu, b >= 0);
            if (fill && b >= 0) fill[w + __popc(in & ((1u << lane) - 1u))] = make_int2(a, b);
            w += __popc(in);
            n += __popc(in);
        }
        if (!fill && lane == 0) cnt[c] = n;
    }
}

// Dense offset -> slot map (entries without a diagonal stay -1).
__global__ void slot_map_kernel(const DiagMeta *__restrict__ meta, int nd, int64_t dmin, int32_t *__restrict__ map) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nd; k += gridDim.x * blockDim.x) map[meta[k].off - dmin] = k;
}

// start[c] = cnt[0] + ... + cnt[c - 1], c = 0 .. n, by one block.
__global__ void __launch_bounds__(1024)
    scan_counts_kernel(const int32_t *__restrict__ cnt, int n, int64_t *__restrict__ start) {
    __shared__ int64_t part[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int64_t carry = 0;
    for (int c0 = 0; c0 < n; c0 += 1024) {
        const int c = c0 + (int)threadIdx.x;
        const int64_t own = c < n ? cnt[c] : 0;
        int64_t v = own;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) part[wid] = v;
        __syncthreads();
        int64_t before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < wid) before += part[w];
            all += part[w];
        }
        if (c < n) start[c] = carry + before + v - own;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) start[n] = carry;
}

// Bits t0 .. t0 + n - 1 (n <= 8) of a mask row of mw words, bits outside it zero; all ones without a mask.
__device__ __forceinline__ uint32_t mask_bits(const uint32_t *__restrict__ row, int64_t mw, int t0, int n) {
    if (!row) return (1u << n) - 1u;
    const int w = t0 >> 5;
    const uint32_t lo = w >= 0 && w < mw ? __ldg(row + w) : 0u, hi = w + 1 >= 0 && w + 1 < mw ? __ldg(row + w + 1) : 0u;
    return __funnelshift_r(lo, hi, t0 & 31) & ((1u << n) - 1u);
}

// A pair that has a nonzero product in a warp's strip of rows: values of row r at A[a + r] and
// B[b + r], rows [lo, hi); the live tiles of the strip (A: V bits per plane) and of the strip's B rows,
// which start `s` rows into a tile (V + 1 bits per plane); its C diagonal, counted from the group's first.
struct __align__(16) LivePair {
    int64_t a, b;
    int32_t lo, hi;
    uint32_t s_c, bits;   // s | C diagonal << 8; bits: A re, A im, B re, B im, a byte each
};
// A C diagonal of the group: value base, rows, first pair.
struct __align__(16) CDiag {
    int64_t base, pstart;
    int32_t lo, hi, pad[2];
};

// (Streaming stores: the products that matter are far larger than L2; 18-qubit H H 1,659 -> 1,597 us.)
template <typename T, int V>
__device__ __forceinline__ void store_rows(T *__restrict__ p, int64_t lo, int64_t hi, int64_t r0, const T (&v)[V]) {
    if (r0 >= lo && r0 + V <= hi) {
        using VT = typename Vec<T, V>::type;
        if constexpr (V == 2)
            __stcs(reinterpret_cast<VT *>(p + r0), VT{v[0], v[1]});
        else
            __stcs(reinterpret_cast<VT *>(p + r0), VT{v[0], v[1], v[2], v[3]});
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i)
            if (r0 + i >= lo && r0 + i < hi) p[r0 + i] = v[i];
    }
}

// Adds the pair's products to the sums of this thread's rows r0 .. r0 + V - 1; all: take both planes
// of both operands whatever the masks say.
template <typename T, int V>
__device__ __forceinline__ void pair_mac(const LivePair &q, bool all, int64_t r0, int lane, const T *__restrict__ Are,
                                         const T *__restrict__ Aim, const T *__restrict__ Bre,
                                         const T *__restrict__ Bim, T (&accr)[V], T (&acci)[V]) {
    // this thread's rows of the pair, if their own tiles are live
    const uint32_t ta = q.bits | q.bits >> 8, tb = (q.bits >> 16) | (q.bits >> 24);
    const int s = (int)(q.s_c & 0xffu) + lane * V;
    if (r0 >= q.hi || r0 + V <= q.lo || !((ta >> (lane * V >> 5)) & 1u) || !(((tb >> (s >> 5)) | (tb >> ((s + V - 1) >> 5))) & 1u))
        return;
    const bool full = r0 >= q.lo && r0 + V <= q.hi;
    auto load = [&](const T *base, bool vec, T(&out)[V]) {
        if (full && vec) {
            load_vec<T, V>(out, base + r0);
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) out[v] = r0 + v >= q.lo && r0 + v < q.hi ? __ldg(base + r0 + v) : (T)0;
        }
    };
    const bool vb = ((q.b + r0) & (V - 1)) == 0;
    const T *pa = Are + q.a, *pai = Aim + q.a, *pb = Bre + q.b, *pbi = Bim + q.b;
    const uint32_t cls = all ? 0xffffffffu : q.bits;
    const bool ar = cls & 0xffu, ai = cls & 0xff00u, br = cls & 0xff0000u, bi = cls & 0xff000000u;
    if (ar != ai && br != bi) {   // one plane each
        T a[V], b[V];
        load(ar ? pa : pai, true, a);
        load(br ? pb : pbi, vb, b);
        if (ar == br) {
#pragma unroll
            for (int v = 0; v < V; ++v) accr[v] = fma(ar ? a[v] : -a[v], b[v], accr[v]);
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) acci[v] = fma(a[v], b[v], acci[v]);
        }
    } else if (ar != ai) {        // one plane of A, both of B
        T a[V], b[V], d[V];
        load(ar ? pa : pai, true, a);
        load(ar ? pb : pbi, vb, b);
        load(ar ? pbi : pb, vb, d);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            accr[v] = fma(ar ? a[v] : -a[v], b[v], accr[v]);
            acci[v] = fma(a[v], d[v], acci[v]);
        }
    } else if (br != bi) {        // both planes of A, one of B
        T a[V], d[V], b[V];
        load(br ? pa : pai, true, a);
        load(br ? pai : pa, true, d);
        load(br ? pb : pbi, vb, b);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            accr[v] = fma(br ? a[v] : -a[v], b[v], accr[v]);
            acci[v] = fma(d[v], b[v], acci[v]);
        }
    } else {
        T xr[V], xi[V], yr[V], yi[V];
        load(pa, true, xr);
        load(pai, true, xi);
        load(pb, vb, yr);
        load(pbi, vb, yi);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            accr[v] = fma(xr[v], yr[v], accr[v]);
            accr[v] = fma(-xi[v], yi[v], accr[v]);
            acci[v] = fma(xr[v], yi[v], acci[v]);
            acci[v] = fma(xi[v], yr[v], acci[v]);
        }
    }
}

// Block (x, y): row strips of x (one per warp, 32 V rows), a run of `chunk` C diagonals of y.  A warp
// takes up to 32 of its C diagonals at a time, and their pairs -- 2.3 per diagonal on the XXZ chain's
// H H, hundreds in a full square -- 32 at a time across the diagonals, a lane per pair: the lane reads
// the pair's metadata and the operands' zero-tile masks of the strip (maskA, maskB: the plane of real
// parts, the plane of imaginary parts psA / psB words behind it) and stages the pair in shared memory
// if its product can hold a nonzero there, so that the chain of dependent reads is paid once for many
// pairs.  The warp then walks the staged pairs, in order, and writes each C diagonal when its pairs
// are done.  A product with a zero factor adds nothing, so a plane that is zero in the strip takes
// part in no product: 1, 2 or 4 multiply-adds per row, each case a body of its own (see
// dia_spmv_kernel).  A diagonal whose sums are not finite is summed again with all four products.
//
// H H of the 18-qubit chain (2.4 GB written, real values): 1,075 -> 677 us, 3.6 TB/s of stores; bound by
// instruction issue (one thread reading its pair's metadata for itself, all four products: 1,075; the
// products by plane alone: 965).  A full complex square of 1,024 rows, 2,047 diagonals: 19.9 -> 8.8 ms,
// 82 % of the FP64 rate (4.3 G multiply-adds).
template <typename T>
__global__ void __launch_bounds__(kSpmvThreads, 4)
    spgemm_numeric_kernel(const DiagMeta *__restrict__ mA, const T *__restrict__ Are, const T *__restrict__ Aim,
                          const DiagMeta *__restrict__ mB, const T *__restrict__ Bre, const T *__restrict__ Bim,
                          const DiagMeta *__restrict__ mC, int ndC, int chunk, const int64_t *__restrict__ pstart,
                          const int2 *__restrict__ pairs, T *__restrict__ Cre, T *__restrict__ Cim,
                          const uint32_t *__restrict__ maskA, int64_t mwA, int64_t psA,
                          const uint32_t *__restrict__ maskB, int64_t mwB, int64_t psB) {
    constexpr int V = VecOf<T>::V;
    __shared__ LivePair sp[kSpmvThreads / 32][32];
    __shared__ CDiag sc[kSpmvThreads / 32][33];
    const int lane = threadIdx.x & 31;
    LivePair *mine = sp[threadIdx.x >> 5];
    CDiag *cd = sc[threadIdx.x >> 5];
    const int64_t w0 = ((int64_t)blockIdx.x * (kSpmvThreads / 32) + (threadIdx.x >> 5)) * 32 * V, r0 = w0 + lane * V;
    const int cend = min(ndC, ((int)blockIdx.y + 1) * chunk);

    // the pair at list position p, staged into L; whether it is live in the strip
    auto stage = [&](int64_t p, int c, int64_t clo, int64_t chi, LivePair &L) {
        const int2 ab = pairs[p];
        const DiagMeta ma = mA[ab.x], mb = mB[ab.y];
        const int64_t lo = max(max(ma.lo, mb.lo - (int64_t)ma.off), clo), hi = min(min(ma.hi, mb.hi - (int64_t)ma.off), chi);
        const int bt = (int)(w0 + ma.off);   // first B row of the strip
        const uint32_t *ka = maskA ? maskA + ab.x * mwA : nullptr, *kb = maskB ? maskB + ab.y * mwB : nullptr;
        const uint32_t ar = mask_bits(ka, mwA, (int)(w0 >> 5), V), ai = mask_bits(ka ? ka + psA : ka, mwA, (int)(w0 >> 5), V);
        const uint32_t br = mask_bits(kb, mwB, bt >> 5, V + 1), bi = mask_bits(kb ? kb + psB : kb, mwB, bt >> 5, V + 1);
        L = LivePair{ma.base, mb.base + ma.off, (int)lo, (int)hi, (uint32_t)(bt & 31) | (uint32_t)c << 8,
                     ar | ai << 8 | br << 16 | bi << 24};
        return w0 < hi && w0 + 32 * V > lo && (ar | ai) && (br | bi);
    };

    for (int c0 = (int)blockIdx.y * chunk; c0 < cend; c0 += 32) {
        const int nc = min(32, cend - c0);
        __syncwarp();
        if (lane < nc) {
            const DiagMeta m = mC[c0 + lane];
            cd[lane] = CDiag{m.base, pstart[c0 + lane], (int)m.lo, (int)m.hi, {0, 0}};
        }
        if (lane == 0) cd[nc].pstart = pstart[c0 + nc];
        __syncwarp();
        T accr[V], acci[V];
#pragma unroll
        for (int v = 0; v < V; ++v) accr[v] = acci[v] = (T)0;
        int c = 0;   // the diagonal being summed
        // write it and go on to the next
        auto finish = [&]() {
            const CDiag q = cd[c];
            if (w0 < q.hi && w0 + 32 * V > q.lo) {
                uint32_t big = 0u, small = ~0u;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    big = max(big, max(abs_hi(accr[v]), abs_hi(acci[v])));
                    small = min(small, min(abs_hi(accr[v]), abs_hi(acci[v])));
                }
                if (maskA && __any_sync(0xffffffffu, unsettled<T>(big, small))) {
#pragma unroll
                    for (int v = 0; v < V; ++v) accr[v] = acci[v] = (T)0;
                    const int64_t p1 = cd[c + 1].pstart;
                    for (int64_t p = q.pstart; p < p1; ++p) {
                        LivePair L;
                        if (stage(p, c, q.lo, q.hi, L)) pair_mac<T, V>(L, true, r0, lane, Are, Aim, Bre, Bim, accr, acci);
                    }
                }
                store_rows<T, V>(Cre + q.base, q.lo, q.hi, r0, accr);
                store_rows<T, V>(Cim + q.base, q.lo, q.hi, r0, acci);
            }
#pragma unroll
            for (int v = 0; v < V; ++v) accr[v] = acci[v] = (T)0;
            ++c;
        };
        const int64_t p1 = cd[nc].pstart;
        for (int64_t p = cd[0].pstart;; p += 32) {
            bool live = false;
            LivePair L;
            if (p + lane < p1) {
                int k = 0;   // the diagonal of pair p + lane: the last one whose list starts at or before it
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (k + step < nc && cd[k + step].pstart <= p + lane) k += step;
                live = stage(p + lane, k, cd[k].lo, cd[k].hi, L);
            }
            const uint32_t set = __ballot_sync(0xffffffffu, live);
            if (live) mine[__popc(set & ((1u << lane) - 1u))] = L;
            __syncwarp();
            const int n = __popc(set), last = p + 32 >= p1;
            for (int k = 0; k < n + last; ++k) {   // after the last pair, the diagonals left
                const int to = k < n ? (int)(mine[k].s_c >> 8) : nc;
                while (c < to) finish();
                if (k < n) pair_mac<T, V>(mine[k], false, r0, lane, Are, Aim, Bre, Bim, accr, acci);
                __syncwarp();
            }
            if (last) break;
            __syncwarp();
        }
    }
}

int spgemm_numeric(const Matrix &A, const Matrix &B, Matrix &C, cudaStream_t s) {
    if (A.prec == DIAQ_C128F2) return set_error(DIAQ_ERR_UNSUPPORTED, "product: convert a c128f2 matrix to c128 first");
    if (A.cols != B.rows || C.rows != A.rows || C.cols != B.cols)
        return set_error(DIAQ_ERR_INVALID, "diaQMatrix product_cuda: dimension mismatch.");
    if (A.prec != B.prec || A.prec != C.prec)
        return set_error(DIAQ_ERR_INVALID, "product: operands must have the same precision");
    C.tmask_ok = false;  // new values
    if (C.nd == 0 || C.rows == 0) return DIAQ_OK;
    const int64_t bmin = -(B.rows - 1), bmax = B.cols - 1;
    const int64_t span = bmax - bmin + 1;
    // scratch: dense offset -> slot map of B, per-C counts, per-C starts
    const size_t mbytes = sizeof(int32_t) * (size_t)span, cbytes = sizeof(int32_t) * (size_t)C.nd,
                 sbytes = sizeof(int64_t) * ((size_t)C.nd + 1);
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    uint8_t *scratch = nullptr;
    DQ_CUDA(dev_malloc_async(&scratch, up(mbytes) + up(cbytes) + sbytes, s));
    int32_t *dmap = (int32_t *)scratch;
    int32_t *dcnt = (int32_t *)(scratch + up(mbytes));
    int64_t *dstart = (int64_t *)(scratch + up(mbytes) + up(cbytes));
    int2 *dpairs = nullptr;
    const int pg = (int)std::max<int64_t>(1, std::min<int64_t>((C.nd + 3) / 4, 8 * num_sms()));
    cudaError_t e = cudaMemsetAsync(dmap, 0xff, mbytes, s);
    if (e == cudaSuccess) {
        slot_map_kernel<<<std::max(1, (B.nd + 255) / 256), 256, 0, s>>>(B.d_meta, B.nd, bmin, dmap);
        spgemm_pairs_kernel<<<pg, 128, 0, s>>>(A.d_meta, A.nd, B.d_meta, dmap, bmin, bmax, C.d_meta, C.nd, dcnt,
                                               nullptr, nullptr);
        scan_counts_kernel<<<1, 1024, 0, s>>>(dcnt, C.nd, dstart);
        e = cudaGetLastError();
    }
    // room for every pair of slots, or -- where that is much -- for as many as there are
    size_t pbytes = sizeof(int2) * (size_t)A.nd * (size_t)B.nd;
    if (pbytes > std::min<size_t>((size_t)64 << 20, alloc_limit())) {
        int64_t npairs = 0;
        if (e == cudaSuccess) e = cudaMemcpyAsync(&npairs, dstart + C.nd, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        pbytes = sizeof(int2) * (size_t)npairs;
    }
    if (e == cudaSuccess) e = dev_malloc_async((void **)&dpairs, std::max<size_t>(pbytes, sizeof(int2)), s);
    if (e == cudaSuccess) {
        spgemm_pairs_kernel<<<pg, 128, 0, s>>>(A.d_meta, A.nd, B.d_meta, dmap, bmin, bmax, C.d_meta, C.nd, nullptr,
                                               dstart, dpairs);
        int64_t maxrows = 1;
        for (const auto &m : C.meta) maxrows = std::max(maxrows, m.hi);
        const int V = A.prec == DIAQ_C128 ? 2 : 4;
        // runs of C diagonals per block: 16 of them (18-qubit H H, whole call: 1,604 us; 32 runs 1,625, 64
        // 1,659, 128 1,735), or more where the rows are few -- some 32 blocks per SM, as the pairs per
        // diagonal vary (1,024 rows, 2,047 diagonals squared: 8.8 ms; 9.4 with half as many runs)
        const unsigned gx = spmv_blocks(maxrows, V);
        const int64_t runs = std::min<int64_t>(C.nd, std::max<int64_t>(16, std::min<int64_t>(65535, 32 * (int64_t)num_sms() / gx)));
        const int chunk = (int)((C.nd + runs - 1) / runs);
        const dim3 grid(gx, (unsigned)((C.nd + chunk - 1) / chunk));
        // the operands' masks (both or neither); taken here, outside any graph capture
        const uint32_t *ka = cached_tile_mask(A, s), *kb = ka ? cached_tile_mask(B, s) : nullptr;
        if (!kb) ka = nullptr;
        const int64_t wa = tile_mask_words(A.rows), wb = tile_mask_words(B.rows), pa = wa * A.nd, pb = wb * B.nd;
        if (ka) {   // the planes of real parts; those of imaginary parts follow
            ka += pa;
            kb += pb;
        }
        if (A.prec == DIAQ_C128)
            spgemm_numeric_kernel<double><<<grid, kSpmvThreads, 0, s>>>(
                A.d_meta, (const double *)A.re, (const double *)A.im, B.d_meta, (const double *)B.re,
                (const double *)B.im, C.d_meta, C.nd, chunk, dstart, dpairs, (double *)C.re, (double *)C.im, ka, wa, pa, kb, wb, pb);
        else
            spgemm_numeric_kernel<float><<<grid, kSpmvThreads, 0, s>>>(
                A.d_meta, (const float *)A.re, (const float *)A.im, B.d_meta, (const float *)B.re,
                (const float *)B.im, C.d_meta, C.nd, chunk, dstart, dpairs, (float *)C.re, (float *)C.im, ka, wa, pa, kb, wb, pb);
        e = cudaGetLastError();
    }
    if (dpairs) cudaFreeAsync(dpairs, s);
    cudaFreeAsync(scratch, s);
    if (e != cudaSuccess) return cuda_status(e, "spgemm numeric", __FILE__, __LINE__);
    return DIAQ_OK;
}

// internal: see Matrix::internal; else the result is the caller's and complete on return.
int spgemm(const Matrix &A, const Matrix &B, bool prune, cudaStream_t s, Matrix **out, bool internal) {
    if (A.prec == DIAQ_C128F2) return set_error(DIAQ_ERR_UNSUPPORTED, "product: convert a c128f2 matrix to c128 first");
    if (A.cols != B.rows) return set_error(DIAQ_ERR_INVALID, "diaQMatrix product_cuda: dimension mismatch.");
    if (A.prec != B.prec) return set_error(DIAQ_ERR_INVALID, "product: operands must have the same precision");
    std::vector<int32_t> offC;
    DQ_TRY(spgemm_symbolic(A, B, offC, s));
    Matrix *C = nullptr;
    // the numeric pass writes every stored value of C: only the gaps around them need zeroing
    DQ_TRY(make_zero(A.rows, B.cols, (int32_t)offC.size(), offC.data(), A.prec, s, &C, false, internal || prune));
    int st = spgemm_numeric(A, B, *C, s);
    if (st == DIAQ_OK) st = zero_gaps(*C, s);
    if (st == DIAQ_OK && prune) st = prune_internal(&C, s);
    if (st == DIAQ_OK && !internal) st = publish(*C);
    if (st == DIAQ_OK && !internal) {
        const cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) st = cuda_status(e, "spgemm", __FILE__, __LINE__);
    }
    if (st != DIAQ_OK) {
        destroy(C);
        return st;
    }
    *out = C;
    return DIAQ_OK;
}

}  // namespace diaq_gb300

using namespace diaq_gb300;

extern "C" {

int diaq_spgemm_symbolic(diaq_matrix_t A, diaq_matrix_t B, int32_t *offsets_out, int32_t *count,
                         void *stream) {
    if (!A || !B || !count) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    std::vector<int32_t> offC;
    DQ_TRY(spgemm_symbolic(*A, *B, offC, (cudaStream_t)stream));
    if (!offC.empty() && !offsets_out) return set_error(DIAQ_ERR_INVALID, "offsets_out is NULL");
    std::copy(offC.begin(), offC.end(), offsets_out);
    *count = (int32_t)offC.size();
    return DIAQ_OK;
}

int diaq_spgemm_numeric(diaq_matrix_t A, diaq_matrix_t B, diaq_matrix_t C, void *stream) {
    if (!A || !B || !C) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    DQ_TRY(spgemm_numeric(*A, *B, *C, (cudaStream_t)stream));
    DQ_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return DIAQ_OK;
}

int diaq_spgemm(diaq_matrix_t A, diaq_matrix_t B, int prune, void *stream, diaq_matrix_t *C) {
    if (!A || !B || !C) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    Matrix *M = nullptr;
    DQ_TRY(spgemm(*A, *B, prune != 0, (cudaStream_t)stream, &M, false));
    *C = handle(M);
    return DIAQ_OK;
}

}  // extern "C"
