// Complex128 SpMV on the FP32 pipes: DIAQ_C128F2 matrices.
//
// GB300 issues FP64 fused multiply-adds at 1/58 of its FP32 rate (0.59 vs 34.6 T/s measured),
// so the float64 SpMV (4 DFMA per stored value) tops out near 2.4 TB/s of matrix traffic -- FP64
// issue, not HBM, bounds it.  A DIAQ_C128F2 matrix keeps 16 bytes per complex value, but each
// float64 v as a pair of floats hi = fl32(v), lo = fl32(v - hi) (a 48-bit significand), and the
// kernel accumulates products of such pairs exactly enough on the FP32 pipes:
//   product   p = ah*xh (+ error fma(ah, xh, -p)) + ah*xl + al*xh          (Dekker/Knuth with FMA)
//   sum       (sh, sl) <- TwoSum(sh, p) with the error and the low parts added to sl
// About 12 FP32 operations per real product-accumulate, 48 per complex value, issued as packed
// two-lane instructions over pairs of rows (24 per complex value and row): ~0.7 T complex values/s
// or more, above the ~0.42 T/s at which HBM delivers the 16-byte values.  Relative error ~1e-14 (2^-48 per value plus accumulation): inside the 1e-12 of
// the float64 path's parity bar.  Range: magnitudes in roughly [1e-30, 1e38] keep the full
// precision (the low float must stay normal).
//
// x arrives as float64 and is split once per call (one pass over N values, without float64
// arithmetic: split64_fast); y is written as float64 (hi + lo in double, 2 conversions and 1 add
// per row).
//
// Storage: the layout of the other precisions, the re (im) array holding the hi plane of
// `capacity` floats followed by the lo plane.
#include <algorithm>

#include "spmv_kernel.cuh"

namespace diaq_gb300 {

__device__ __forceinline__ void split64(double v, float &h, float &l) {
    h = (float)v;
    l = (float)(v - (double)h);
}

// split64 kept out of line, for the rare values split64_fast leaves to it.  Inlined, its
// conversions and float64 subtraction are if-converted into the fast path and issue on GB300's
// FP64 pipe for every value, taken or not: the split of x took 18.5 us instead of 8.2.
__device__ __noinline__ void split64_outlined(double v, float &h, float &l) { split64(v, h, l); }

// The split of x with bit operations and float32 arithmetic only.  hi is v truncated to 24
// significant bits (the high word and 3 bits of the low one); lo is the remaining 29 bits ml,
// rounded to 24 bits as 64 a + c (a = ml >> 6 and c = ml & 63 made exact floats by the 2^23
// magic number, one rounding in the fma) and scaled by v's exponent through its exponent field:
// |v - hi - lo| <= 2^-48 |v|, split64's bound.  Exponents where hi or lo would not be a normal
// float (|v| outside about [1e-22, 3e38]) take split64.
__device__ __forceinline__ void split64_fast(double v, float &h, float &l) {
    const uint32_t H = (uint32_t)__double2hiint(v), L = (uint32_t)__double2loint(v);
    const uint32_t e = (H >> 20) & 0x7ffu;
    if (e < 950u || e > 1150u) {
        split64_outlined(v, h, l);
        return;
    }
    const uint32_t sign = H & 0x80000000u;
    h = __uint_as_float(sign | ((e - 896u) << 23) | ((H & 0xfffffu) << 3) | (L >> 29));
    const uint32_t ml = L & 0x1fffffffu;  // lo = ml * 2^(e - 1075), ml < 2^29
    const float fa = __fsub_rn(__uint_as_float(0x4b000000u | (ml >> 6)), 8388608.0f);
    const float fc = __fsub_rn(__uint_as_float(0x4b000000u | (ml & 63u)), 8388608.0f);
    const float f = __fmaf_rn(fa, 64.0f, fc);
    l = ml ? __uint_as_float(sign | (__float_as_uint(f) - ((1075u - e) << 23))) : __uint_as_float(sign);
}

// packed float64 -> hi/lo planes
__global__ void f2_scatter_kernel(const DiagMeta *__restrict__ meta, int nd, const double *__restrict__ sre,
                                  const double *__restrict__ sim, float *__restrict__ re, float *__restrict__ im,
                                  int64_t cap) {
    for (int k = blockIdx.y; k < nd; k += gridDim.y) {
        const DiagMeta m = meta[k];
        const int64_t len = m.hi - m.lo;
        for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < len; j += (int64_t)gridDim.x * blockDim.x) {
            const int64_t d = m.base + m.lo + j;
            split64(sre[m.pstart + j], re[d], re[cap + d]);
            split64(sim[m.pstart + j], im[d], im[cap + d]);
        }
    }
}

// hi/lo planes -> packed float64
__global__ void f2_gather_kernel(const DiagMeta *__restrict__ meta, int nd, const float *__restrict__ re,
                                 const float *__restrict__ im, int64_t cap, double *__restrict__ dre,
                                 double *__restrict__ dim) {
    for (int k = blockIdx.y; k < nd; k += gridDim.y) {
        const DiagMeta m = meta[k];
        const int64_t len = m.hi - m.lo;
        for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < len; j += (int64_t)gridDim.x * blockDim.x) {
            const int64_t s = m.base + m.lo + j;
            dre[m.pstart + j] = (double)re[s] + (double)re[cap + s];
            dim[m.pstart + j] = (double)im[s] + (double)im[cap + s];
        }
    }
}

// both float64 vectors of state blockIdx.y -> their four hi/lo planes in one launch; vec: every
// state's x_re and x_im are 16-byte aligned, so pairs of values move as double2 -> float2.  State q reads
// at q * ldx and writes at q * 4 np (planes re hi, re lo, im hi, im lo of np values).
__global__ void f2_split_pair_kernel(const double *__restrict__ xr, const double *__restrict__ xi, int64_t n, int64_t ldx,
                                     int vec, float *__restrict__ planes, int64_t np) {
    xr += blockIdx.y * ldx;
    xi += blockIdx.y * ldx;
    float *rh = planes + blockIdx.y * 4 * np, *rl = rh + np, *ih = rl + np, *il = ih + np;
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    int64_t done = 0;
    if (vec) {
        const int64_t n2 = n / 2;
        for (int64_t i = t0; i < n2; i += stride) {
            const double2 a = reinterpret_cast<const double2 *>(xr)[i], b = reinterpret_cast<const double2 *>(xi)[i];
            float h0, l0, h1, l1;
            split64_fast(a.x, h0, l0);
            split64_fast(a.y, h1, l1);
            reinterpret_cast<float2 *>(rh)[i] = make_float2(h0, h1);
            reinterpret_cast<float2 *>(rl)[i] = make_float2(l0, l1);
            split64_fast(b.x, h0, l0);
            split64_fast(b.y, h1, l1);
            reinterpret_cast<float2 *>(ih)[i] = make_float2(h0, h1);
            reinterpret_cast<float2 *>(il)[i] = make_float2(l0, l1);
        }
        done = 2 * n2;
    }
    for (int64_t i = done + t0; i < n; i += stride) {
        split64_fast(xr[i], rh[i], rl[i]);
        split64_fast(xi[i], ih[i], il[i]);
    }
}

// s += a*x for float pairs (see the file comment), two rows at once: TwoProd (ph + the exact
// remainder by FMA) and TwoSum, on the packed two-lane FP32 instructions (__fmul2_rn, __ffma2_rn,
// __fadd2_rn: each lane the scalar operation with its rounding; a - b as a + (-b), which is exact).
// The _rn intrinsics keep the compiler from fusing the product into the sum, which would break
// both identities.  Negate ah and al to subtract.  Against one row per instruction: 101.1 -> 99.5
// us per SpMV on the 20-qubit chain, the same bits.
struct F2P {
    float2 h, l;
};
__device__ __forceinline__ float2 neg2(float2 v) { return make_float2(-v.x, -v.y); }
__device__ __forceinline__ void f2_mac2(F2P &s, float2 ah, float2 al, float2 xh, float2 xl) {
    const float2 ph = __fmul2_rn(ah, xh);
    float2 pl = __ffma2_rn(ah, xh, neg2(ph));
    pl = __ffma2_rn(ah, xl, pl);
    pl = __ffma2_rn(al, xh, pl);
    const float2 t = __fadd2_rn(s.h, ph);
    const float2 bb = __fadd2_rn(t, neg2(s.h));
    const float2 e = __fadd2_rn(__fadd2_rn(s.h, neg2(__fadd2_rn(t, neg2(bb)))), __fadd2_rn(ph, neg2(bb)));
    s.h = t;
    s.l = __fadd2_rn(s.l, __fadd2_rn(e, pl));
}

// y = A x: each thread owns VR = 4 consecutive rows; hi and lo planes are separate SoA arrays, so
// every matrix load is a 16-byte vector of 4 rows.  Strips that lie inside a diagonal read the
// four x planes as aligned vectors shifted across lanes (the x planes are this file's scratch,
// padded to a multiple of 32 values, so the aligned vectors stay inside them; values past column
// cols are read but never used).  Each diagonal's offset, row range and the block's mask word are
// staged as one 16-byte shared-memory record.  (Prefetching the warp's strip of the four matrix
// planes into L2 a few diagonals ahead measured slower on the 20-qubit XXZ chain, 216 against
// 194 us, and was dropped.)

// The chunk of diagonals staged in sq / sb added to a thread's four rows (two F2P row pairs per
// accumulator).  IM = false: the matrix holds no imaginary part, half the loads and half the products.
template <bool IM>
__device__ __forceinline__ void f2_accumulate(const int4 *sq, const int64_t *sb, int cn, int64_t r0, int lane,
                                              const float *__restrict__ are, const float *__restrict__ aim, int64_t cap,
                                              int64_t rows, const float *__restrict__ xrh,
                                              const float *__restrict__ xrl, const float *__restrict__ xih,
                                              const float *__restrict__ xil, F2P (&sr)[2], F2P (&si)[2]) {
    constexpr int V = 4;
    const int64_t w0 = r0 - (int64_t)V * lane;
    const int wbit = (int)((w0 >> 5) & 31);  // the warp's 128 rows: 4 tiles, bits wbit .. wbit + 3
    for (int k = 0; k < cn; ++k) {
        const int4 q = sq[k];
        const int64_t lo = q.y, hi = q.z;
        const uint32_t mword = (uint32_t)q.w;
        // the same for the whole warp (the windows below are shuffled across its lanes)
        if (w0 >= hi || w0 + 32 * V <= lo || !((mword >> wbit) & 0xfu)) continue;
        const int64_t b = sb[k] + r0, c = r0 + q.x;
        float arh[V], arl[V], aih[V], ail[V];
        float xrhv[V], xrlv[V], xihv[V], xilv[V];
        if (w0 >= lo && w0 + 32 * V <= hi) {
            // an aligned window needs no shuffle: a lane whose tile is zero drops out alone
            if ((q.x & 3) == 0 && !((mword >> ((r0 >> 5) & 31)) & 1u)) continue;
            load_vec_stream<float, V>(arh, are + b);
            load_vec_stream<float, V>(arl, are + cap + b);
            if constexpr (IM) {
                load_vec_stream<float, V>(aih, aim + b);
                load_vec_stream<float, V>(ail, aim + cap + b);
            }
            const int s = (int)(c & 3);
            const int64_t ca = c - s;
            shifted_window(xrhv, xrh + ca, s, lane);
            shifted_window(xrlv, xrl + ca, s, lane);
            shifted_window(xihv, xih + ca, s, lane);
            shifted_window(xilv, xil + ca, s, lane);
        } else {
            if (r0 >= rows || r0 + V <= lo || r0 >= hi) continue;
            load_vec_stream<float, V>(arh, are + b);
            load_vec_stream<float, V>(arl, are + cap + b);
            if constexpr (IM) {
                load_vec_stream<float, V>(aih, aim + b);
                load_vec_stream<float, V>(ail, aim + cap + b);
            }
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const bool ok = (r0 + v >= lo) && (r0 + v < hi);
                xrhv[v] = ok ? __ldg(xrh + c + v) : 0.f;
                xrlv[v] = ok ? __ldg(xrl + c + v) : 0.f;
                xihv[v] = ok ? __ldg(xih + c + v) : 0.f;
                xilv[v] = ok ? __ldg(xil + c + v) : 0.f;
                if (!ok) arh[v] = arl[v] = 0.f;
                if (IM && !ok) aih[v] = ail[v] = 0.f;
            }
        }
#pragma unroll
        for (int v = 0; v < V; v += 2) {
            const float2 rh = make_float2(arh[v], arh[v + 1]), rl = make_float2(arl[v], arl[v + 1]);
            const float2 xrh2 = make_float2(xrhv[v], xrhv[v + 1]), xrl2 = make_float2(xrlv[v], xrlv[v + 1]);
            const float2 xih2 = make_float2(xihv[v], xihv[v + 1]), xil2 = make_float2(xilv[v], xilv[v + 1]);
            if constexpr (IM) {
                const float2 ih = make_float2(aih[v], aih[v + 1]), il = make_float2(ail[v], ail[v + 1]);
                f2_mac2(sr[v / 2], rh, rl, xrh2, xrl2);
                f2_mac2(sr[v / 2], neg2(ih), neg2(il), xih2, xil2);
                f2_mac2(si[v / 2], rh, rl, xih2, xil2);
                f2_mac2(si[v / 2], ih, il, xrh2, xrl2);
            } else {
                f2_mac2(sr[v / 2], rh, rl, xrh2, xrl2);
                f2_mac2(si[v / 2], rh, rl, xih2, xil2);
            }
        }
    }
}

// Whether a thread's sums have to be taken again in full (see unsettled; a NaN high part makes its low
// part NaN).
template <int N>
__device__ __forceinline__ bool f2_unsettled(const F2P (&a)[N], const F2P (&b)[N]) {
    uint32_t big = 0u, small = ~0u;
#pragma unroll
    for (int v = 0; v < N; ++v) {
        const uint32_t h[4] = {abs_hi(a[v].h.x), abs_hi(a[v].h.y), abs_hi(b[v].h.x), abs_hi(b[v].h.y)};
        const uint32_t l[4] = {abs_hi(a[v].l.x), abs_hi(a[v].l.y), abs_hi(b[v].l.x), abs_hi(b[v].l.y)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            big = max(big, max(h[i], l[i]));
            small = min(small, h[i]);
        }
    }
    return unsettled<float>(big, small);
}

// State blockIdx.y: x planes at y * 4 np, y at y * ldy.  REAL: the matrix holds no imaginary part (and
// one chunk of metadata), half the loads and products; a warp whose sums are not finite sums again in
// full, as the products left out would have spread an infinite or NaN x.  20-qubit chain: 100 -> 82 us.
template <int MINB, bool REAL>
__global__ void __launch_bounds__(kSpmvThreads, MINB)
    f2_spmv_kernel(const DiagMeta *__restrict__ meta, int nd, const float *__restrict__ are,
                   const float *__restrict__ aim, int64_t cap, int64_t rows, const float *__restrict__ planes, int64_t np,
                   double *__restrict__ yr, double *__restrict__ yi, int64_t ldy, const uint32_t *__restrict__ tmask,
                   int64_t mw) {
    constexpr int V = 4;
    __shared__ int4 sq[kMetaChunk];     // offset, lo, hi, mask word (the block's 1024 rows are one word)
    __shared__ int64_t sb[kMetaChunk];  // value base
    const int lane = threadIdx.x & 31;
    const int64_t r0 = ((int64_t)blockIdx.x * kSpmvThreads + threadIdx.x) * V;
    const int64_t w0 = r0 - (int64_t)V * lane;
    const float *xrh = planes + blockIdx.y * 4 * np, *xrl = xrh + np, *xih = xrl + np, *xil = xih + np;
    F2P sr[V / 2], si[V / 2];   // rows (0, 1) and (2, 3)
    auto clear = [&]() {
#pragma unroll
        for (int v = 0; v < V / 2; ++v) sr[v] = si[v] = F2P{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    };
    clear();
    for (int c0 = 0; c0 < nd; c0 += kMetaChunk) {
        const int cn = min(kMetaChunk, nd - c0);
        __syncthreads();
        for (int i = threadIdx.x; i < cn; i += kSpmvThreads) {
            const DiagMeta m = meta[c0 + i];
            const uint32_t w = tmask ? tmask[(int64_t)(c0 + i) * mw + blockIdx.x] : 0xffffffffu;
            sq[i] = make_int4(m.off, (int)m.lo, (int)m.hi, (int)w);
            sb[i] = m.base;
        }
        __syncthreads();
        if (w0 >= rows) continue;
        if constexpr (REAL) {
            f2_accumulate<false>(sq, sb, cn, r0, lane, are, aim, cap, rows, xrh, xrl, xih, xil, sr, si);
            if (!__any_sync(0xffffffffu, f2_unsettled(sr, si))) continue;
            clear();
        }
        f2_accumulate<true>(sq, sb, cn, r0, lane, are, aim, cap, rows, xrh, xrl, xih, xil, sr, si);
    }
    if (r0 >= rows) return;
    yr += blockIdx.y * ldy;
    yi += blockIdx.y * ldy;
#pragma unroll
    for (int v = 0; v < V; ++v)
        if (r0 + v < rows) {
            const F2P &a = sr[v / 2], &b = si[v / 2];
            yr[r0 + v] = (double)((v & 1) ? a.h.y : a.h.x) + (double)((v & 1) ? a.l.y : a.l.x);
            yi[r0 + v] = (double)((v & 1) ? b.h.y : b.h.x) + (double)((v & 1) ? b.l.y : b.l.x);
        }
}

// The real and imaginary sum of one row, in the two lanes of packed instructions: the arithmetic (and
// the bits) of f2_mac2.  (re, im) += (ah, al) * (x, y)
struct F2Row {
    float2 h, l;
};
__device__ __forceinline__ void f2_mac_row(F2Row &s, float2 ah, float2 al, float2 xh, float2 xl) {
    F2P t{s.h, s.l};
    f2_mac2(t, ah, al, xh, xl);
    s = F2Row{t.h, t.l};
}

// One row per thread in blocks of 64, for few rows x states (see dia_spmv_row_kernel): ballots find the
// diagonals that hold a real or an imaginary nonzero in the warp's 32 rows, the loads of U of them are
// issued together, and a plane that is zero there takes part in no product; a warp whose sums are not
// finite sums again in full.  Against f2_spmv_kernel, split included: 12-qubit chain 12.3 us (24.3),
// 16-qubit Pauli sum 25.9 (74.3), 250,007 rows of 37 diagonals 35.9 (54.4), 8 states of 100,001 rows 51.3
// (57.7).  The lines, in rows x states of a launch: a matrix without an imaginary part costs the other
// kernel half, so from some 360,000 on four rows per thread are the better form (16-qubit chain, 5
// states, 327,680: 32.8 us against 34.9; 17 qubits, 3 states, 393,216: Ising 45.2 against 42.0, XXZ 36.9 and
// 37.0; 524,288: 50 against 46) -- but where its blocks are a little more than run at a time (four per SM)
// their last wave is mostly empty (655,360: Ising 69 against 73) -- a complex one from some 900,000 on
// (Pauli sum, 786,432: 144 against 162; 917,504: 159 against 150; bands of 850,000 57 against 66, of
// 1,040,000 68 against 71).
constexpr int64_t kF2RowKernelMax = 900000, kF2RowKernelMaxReal = 360000;
inline bool f2_row_kernel_pays(int64_t rows, int states, bool real) {
    if (!real) return rows * states <= kF2RowKernelMax;
    const int64_t blocks = spmv_blocks(rows, 4) * (int64_t)states, wave = 4 * (int64_t)num_sms();
    return rows * states <= kF2RowKernelMaxReal || (blocks > wave && 5 * blocks < 6 * wave);
}
template <int U>
__global__ void __launch_bounds__(64)
    f2_spmv_row_kernel(const DiagMeta *__restrict__ meta, int nd, const float *__restrict__ are,
                       const float *__restrict__ aim, int64_t cap, int rows, const float *__restrict__ planes, int64_t np,
                       double *__restrict__ yr, double *__restrict__ yi, int64_t ldy, const uint32_t *__restrict__ tmask,
                       int64_t mw) {
    const int lane = (int)threadIdx.x & 31, r = (int)(blockIdx.x * 64 + threadIdx.x), w0 = r - lane;
    if (w0 >= rows) return;
    const float *xrh = planes + blockIdx.y * 4 * np + r, *xrl = xrh + np, *xih = xrl + np, *xil = xih + np;
    const float *arh = are + r, *aih = aim + r;
    F2Row acc;
    for (int pass = 0;; ++pass) {
        acc = F2Row{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        for (int c0 = 0; c0 < nd; c0 += 32) {
            int off = 0, lo = 0, hi = 0;
            int64_t base = 0;
            bool re = false, im = false;
            if (c0 + lane < nd) {
                const DiagMeta m = meta[c0 + lane];
                off = m.off;
                lo = (int)m.lo;
                hi = (int)m.hi;
                base = m.base;
                if (w0 < hi && w0 + 32 > lo) {
                    const int64_t at = (int64_t)(c0 + lane) * mw + (w0 >> 10);
                    re = !tmask || (tmask[nd * mw + at] >> ((w0 >> 5) & 31)) & 1u;
                    im = !tmask || (tmask[2 * nd * mw + at] >> ((w0 >> 5) & 31)) & 1u;
                }
            }
            uint32_t mr = __ballot_sync(0xffffffffu, re), mi = __ballot_sync(0xffffffffu, im), live = mr | mi;
            if (pass) mr = mi = live;
            while (live) {
                float ah[U], al[U], bh[U], bl[U];
                float2 xh[U], xl[U];
                uint32_t bit[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    bit[u] = live & (0u - live);
                    const int j = live ? __ffs(live) - 1 : 0;
                    live &= live - 1u;
                    const int o = __shfl_sync(0xffffffffu, off, j), l = __shfl_sync(0xffffffffu, lo, j),
                              h = __shfl_sync(0xffffffffu, hi, j);
                    const int64_t b = __shfl_sync(0xffffffffu, base, j);
                    const bool in = bit[u] && r >= l && r < h, inr = in && (mr & bit[u]), ini = in && (mi & bit[u]);
                    ah[u] = inr ? __ldcs(arh + b) : 0.f;
                    al[u] = inr ? __ldcs(arh + cap + b) : 0.f;
                    bh[u] = ini ? __ldcs(aih + b) : 0.f;
                    bl[u] = ini ? __ldcs(aih + cap + b) : 0.f;
                    xh[u] = make_float2(in ? __ldg(xrh + o) : 0.f, in ? __ldg(xih + o) : 0.f);
                    xl[u] = make_float2(in ? __ldg(xrl + o) : 0.f, in ? __ldg(xil + o) : 0.f);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (mr & bit[u]) f2_mac_row(acc, make_float2(ah[u], ah[u]), make_float2(al[u], al[u]), xh[u], xl[u]);
                    if (mi & bit[u])   // re -= b y, im += b x
                        f2_mac_row(acc, make_float2(-bh[u], bh[u]), make_float2(-bl[u], bl[u]),
                                   make_float2(xh[u].y, xh[u].x), make_float2(xl[u].y, xl[u].x));
                }
            }
        }
        if (pass || !tmask) break;
        const uint32_t big = max(max(abs_hi(acc.h.x), abs_hi(acc.h.y)), max(abs_hi(acc.l.x), abs_hi(acc.l.y)));
        const uint32_t small = min(abs_hi(acc.h.x), abs_hi(acc.h.y));
        if (!__any_sync(0xffffffffu, unsettled<float>(big, small))) break;
    }
    if (r >= rows) return;
    yr[blockIdx.y * ldy + r] = (double)acc.h.x + (double)acc.l.x;
    yi[blockIdx.y * ldy + r] = (double)acc.h.y + (double)acc.l.y;
}

__global__ void f2_from_c128_kernel(const DiagMeta *__restrict__ meta, int nd, const double *__restrict__ sre,
                                    const double *__restrict__ sim, float *__restrict__ re, float *__restrict__ im,
                                    int64_t cap) {
    for (int k = blockIdx.y; k < nd; k += gridDim.y) {
        const DiagMeta m = meta[k];
        for (int64_t r = m.lo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m.hi; r += (int64_t)gridDim.x * blockDim.x) {
            split64(sre[m.base + r], re[m.base + r], re[cap + m.base + r]);
            split64(sim[m.base + r], im[m.base + r], im[cap + m.base + r]);
        }
    }
}

__global__ void c128_from_f2_kernel(const DiagMeta *__restrict__ meta, int nd, const float *__restrict__ re,
                                    const float *__restrict__ im, int64_t cap, double *__restrict__ dre,
                                    double *__restrict__ dim) {
    for (int k = blockIdx.y; k < nd; k += gridDim.y) {
        const DiagMeta m = meta[k];
        for (int64_t r = m.lo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m.hi; r += (int64_t)gridDim.x * blockDim.x) {
            dre[m.base + r] = (double)re[m.base + r] + (double)re[cap + m.base + r];
            dim[m.base + r] = (double)im[m.base + r] + (double)im[cap + m.base + r];
        }
    }
}

static dim3 f2_grid(const Matrix &M) {
    int64_t maxlen = 1;
    for (const auto &m : M.meta) maxlen = std::max(maxlen, m.hi - m.lo);
    return dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>((maxlen + 1023) / 1024, 4 * num_sms())),
                (unsigned)std::min<int64_t>(std::max<int32_t>(M.nd, 1), 65535));
}

int f2_scatter(Matrix &M, const double *re, const double *im, cudaStream_t s) {
    M.tmask_ok = false;
    if (M.nd == 0) return DIAQ_OK;
    f2_scatter_kernel<<<f2_grid(M), 256, 0, s>>>(M.d_meta, M.nd, re, im, (float *)M.re, (float *)M.im, M.capacity);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

int f2_gather(const Matrix &M, double *re, double *im, cudaStream_t s) {
    if (M.nd == 0) return DIAQ_OK;
    f2_gather_kernel<<<f2_grid(M), 256, 0, s>>>(M.d_meta, M.nd, (const float *)M.re, (const float *)M.im, M.capacity, re,
                                                im);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

// Same offsets and layout (src and dst planned alike); one precision is C128, the other C128F2.
int f2_convert(const Matrix &src, Matrix &dst, cudaStream_t s) {
    dst.tmask_ok = false;
    if (dst.nd == 0) return DIAQ_OK;
    if (src.prec == DIAQ_C128 && dst.prec == DIAQ_C128F2)
        f2_from_c128_kernel<<<f2_grid(dst), 256, 0, s>>>(src.d_meta, src.nd, (const double *)src.re, (const double *)src.im,
                                                        (float *)dst.re, (float *)dst.im, dst.capacity);
    else if (src.prec == DIAQ_C128F2 && dst.prec == DIAQ_C128)
        c128_from_f2_kernel<<<f2_grid(dst), 256, 0, s>>>(src.d_meta, src.nd, (const float *)src.re, (const float *)src.im,
                                                        src.capacity, (double *)dst.re, (double *)dst.im);
    else
        return set_error(DIAQ_ERR_UNSUPPORTED, "c128f2 matrices convert to and from c128 only");
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

int f2_spmv(const Matrix &A, int nrhs, const double *xr, const double *xi, int64_t ldx, double *yr, double *yi,
            int64_t ldy, cudaStream_t s) {
    if (A.rows == 0 || nrhs <= 0) return DIAQ_OK;
    const int64_t n = A.cols;
    const int64_t np = std::max<int64_t>((n + 31) / 32 * 32, 32);  // planes 128-byte aligned: equal alignment for hi and lo
    // up to 8 states per launch; one, if their planes do not fit
    int k = std::min(nrhs, 8);
    float *buf = nullptr;
    cudaError_t e = dev_malloc_async(&buf, sizeof(float) * 4 * (size_t)np * (size_t)k, s);
    if (e == cudaErrorMemoryAllocation && k > 1) {
        cudaGetLastError();
        k = 1;
        e = dev_malloc_async(&buf, sizeof(float) * 4 * (size_t)np, s);
    }
    if (e != cudaSuccess) return cuda_status(e, "f2 spmv workspace", __FILE__, __LINE__);
    const uint32_t *tmask = cached_tile_mask(A, s);
    const float *are = (const float *)A.re, *aim = (const float *)A.im;
    const int64_t mw = tile_mask_words(A.rows);
    const bool real = tmask && A.real && A.nd <= kMetaChunk;
    for (int q = 0; q < nrhs; q += k) {
        const int kq = std::min(k, nrhs - q);
        const double *pr = xr + q * ldx, *pi = xi + q * ldx;
        double *qr = yr + q * ldy, *qi = yi + q * ldy;
        const dim3 g((unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 8 * num_sms() / kq + 1)), (unsigned)kq);
        const int vec = ((uintptr_t)pr % 16 == 0) && ((uintptr_t)pi % 16 == 0) && (kq == 1 || ldx % 2 == 0);
        f2_split_pair_kernel<<<g, 256, 0, s>>>(pr, pi, n, ldx, vec, buf, np);
        if (f2_row_kernel_pays(A.rows, kq, real)) {
            f2_spmv_row_kernel<4><<<dim3((unsigned)((A.rows + 63) / 64), (unsigned)kq), 64, 0, s>>>(
                A.d_meta, A.nd, are, aim, A.capacity, (int)A.rows, buf, np, qr, qi, ldy, tmask, mw);
        } else {
            // four blocks per SM (64 registers): 82 us on the 20-qubit chain; three (78 registers) 90, five
            // and six spill (110, 134)
            auto go = [&](auto kernel) {
                kernel<<<dim3(spmv_blocks(A.rows, 4), (unsigned)kq), kSpmvThreads, 0, s>>>(
                    A.d_meta, A.nd, are, aim, A.capacity, A.rows, buf, np, qr, qi, ldy, tmask, mw);
            };
            if (real) go(f2_spmv_kernel<4, true>);
            else go(f2_spmv_kernel<4, false>);
        }
    }
    e = cudaGetLastError();
    cudaFreeAsync(buf, s);
    if (e != cudaSuccess) return cuda_status(e, "f2 spmv", __FILE__, __LINE__);
    return DIAQ_OK;
}

}  // namespace diaq_gb300
