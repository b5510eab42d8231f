// Conversions to float pairs without FP64 instructions, and row sums with the
// vectors across the lanes, for the float-instruction sparse kernels
// (csrc/spmv_lp.cu, csrc/expm_lp.cu, csrc/expm_vl.cu).
#pragma once
#include <type_traits>
#include "lp_modes.cuh"

namespace {

// The pair of x 2^-k rounded to nearest, bit for bit pf_from_double(x 2^-k):
// the high part is the top 24 significant bits rounded, the low part the signed
// rest (at most 2^28 units of x's last place) as an integer conversion and a
// multiplication by a power of two.  One conversion instruction and no FP64:
// the FP64 form takes five, at a sixty-fourth of the integer rate.  Zeros are
// their own pair; values whose low part would leave the normal float range
// (and infinities and NaN) take the FP64 form.
__device__ __forceinline__ pf pair_rn_scaled(double x, int k)
{
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const int E = (int)((hi >> 20) & 0x7ffu), ef = E - 896 - k;
    if (E == 0 || E == 0x7ff || (unsigned)(ef - 54) >= 200u) {
        if (((hi << 1) | lo) == 0u) return pf{__uint_as_float(hi), 0.f};
        return pf_from_double(x * pow2(-k));
    }
    const uint32_t rest = lo & 0x1fffffffu;
    const bool up = rest + ((lo >> 29) & 1u) > 0x10000000u;      // to nearest, ties to even
    const uint32_t h = ((hi & 0x80000000u) | ((uint32_t)ef << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29)) + (up ? 1u : 0u);
    int r = (int)rest - (up ? 0x20000000 : 0);
    if (hi & 0x80000000u) r = -r;
    return pf{__uint_as_float(h), __fmul_rn(__int2float_rn(r), __uint_as_float((uint32_t)(ef - 52) << 23))};
}

// x 2^-k in the storage of a mode
template <class M> __device__ __forceinline__ typename M::S scaled_from_double(double x, int k);
template <> __device__ __forceinline__ pf scaled_from_double<ModePF>(double x, int k) { return pair_rn_scaled(x, k); }
template <> __device__ __forceinline__ float scaled_from_double<ModeF32>(double x, int k) { return (float)(x * pow2(-k)); }

__device__ __forceinline__ pf shfl_pair(pf a, int src)
{
    return pf{__shfl_sync(0xffffffffu, a.h, src & 31), __shfl_sync(0xffffffffu, a.l, src & 31)};
}

// real value times real x
template <class M>
__device__ __forceinline__ void rmul_acc(typename M::S &ar, typename M::S &, typename M::S d, typename M::S x)
{
    M::fma(ar, d, x);
}
// complex value times real x
template <class M>
__device__ __forceinline__ void rmul_acc(typename M::S &ar, typename M::S &ai, const cx<typename M::S> &d,
                                         typename M::S x)
{
    M::fma(ar, d.re, x);
    M::fma(ai, d.im, x);
}

// Lane groups of the many-vector kernels: VL lanes walk a row, or one of
// `split` interleaved parts of a long one; 32 / (VL split) rows to a warp;
// lanes left over own none.  The vectors are swept at most eight at a time in
// sweeps of equal width, so few lanes go without one (13 vectors: two sweeps
// of 7).
static inline int vl_lanes(int64_t nvec)
{
    const int64_t sweeps = (nvec + 7) / 8;
    return (int)((nvec + sweeps - 1) / sweeps);
}

// Parts of a row: a power of two that fits a warp.  Two reasons to divide it.
// Few vectors: 16 rows to a warp read 16 far places of the words at once, so two
// vectors take a part per 32 entries, three to five two parts from 64 or 128
// entries (a float-pair product of 2 vectors, 60 k rows of 128 entries: 66 us in
// one part, 50 in four; a term 64 and 49).  Few rows: parts of at least 16
// entries while there are less than `lanes` lanes at work (8 vectors, 1000 rows
// of 1000 entries: a product 109 -> 40 us, a term 97 -> 34; 300 rows of 300, 36
// -> 18).  Beyond either it costs: at 60 k rows of 64 entries and 8 vectors a term
// takes 67 us in one part, 81 in two.
static inline int vl_split(int64_t n, int64_t nnz, int VL, int64_t lanes = 100000)
{
    const int64_t avg = n > 0 ? nnz / n : 0;
    int s = 1;
    while (2 * s * VL <= 32) {
        const bool longs = VL == 2 ? avg >= 64 * s : VL <= 5 && s == 1 && avg >= (VL == 3 ? 64 : 128);
        if (!longs && !(avg >= 32 * s && 2 * s * VL * n <= lanes)) break;
        s *= 2;
    }
    return s;
}

constexpr int VB = 4;      // nonzeros of a row in flight

// Chains of a row's sum in one lane, places taken in turn: two, as two lanes of
// a row hand-out.  Long rows of plain floats take four, summed every VFLUSH
// batches, since their roundings are what a result is made of: RMS error of a
// complex64 product of 8 vectors, rows of 100 and 400 entries, 1.8e-7 and 3.6e-7 with
// two chains, 8.1e-8 and 9.4e-8 so (row hand-out, 4 and 32 lanes: 1.0e-7 and
// 1.1e-7).  Four for short rows cost 13% (200 k rows of 20, 32.7 -> 37.1 us), and for
// float pairs spills (45.3 -> 47.6 us, the L = 20 Ising sector).
template <class M, bool LONG> constexpr int VCHAINS = LONG && std::is_same<M, ModeF32>::value ? 4 : 2;
constexpr int VFLUSH = 4;

// Whether an operand takes the kernels for long rows: parts of a row, sweeps in
// blocks of their own, sums taken now and then.  Their arithmetic costs the others
// 2 to 5% (a term of 8 vectors, 200 k rows of 20).
template <class M>
static inline bool vl_long(int64_t n, int64_t nnz, int split)
{
    return split > 1 || (std::is_same<M, ModeF32>::value && n > 0 && nnz / n >= 32);
}

// A lane's place in its warp: vector v of part `part` of row `grp` of `rows`;
// lane0: the first lane of its VL.
struct VlPlace {
    int rows, grp, part, v, lane0;
};
__device__ __forceinline__ VlPlace vl_place(int VL, int split)
{
    const int lane = threadIdx.x & 31, per = VL * split, grp = lane / per, in = lane - grp * per;
    const int part = split == 1 ? 0 : in / VL;
    const int v = in - part * VL;
    return {32 / per, grp, part, v, lane - v};
}

// One batch of VB nonzeros of a row for one vector, the column words in cur
// (WPL per lane of the group, whose first lane is lane0), entry k the first.
// FULL: all of them belong to the row; otherwise only the first `left`.  A
// word past the row's end is zero and its gather reads column 0: an address
// without a predicate, its product is skipped.
template <class M, class DV, bool XC, class IT, int VMODE, int WPL, bool FULL, class ST, int NC>
__device__ __forceinline__ void vl_batch(const uint32_t (&cur)[WPL], int lane0, const DV *__restrict__ data,
                                         const uint8_t *__restrict__ codes, const DV *tab,
                                         const char *__restrict__ x, ST stride, IT k, int left,
                                         typename M::S (&ar)[NC], typename M::S (&ai)[NC])
{
    using XE = typename std::conditional<XC, typename M::BE, typename M::S>::type;
    XE xe[VB];
    DV d[VB];
#pragma unroll
    for (int u = 0; u < VB; u++) {
        const uint32_t w = __shfl_sync(0xffffffffu, cur[u % WPL], lane0 + u / WPL);
        if constexpr (VMODE == 2) d[u] = tab[w & 255u];
        const XE *p = reinterpret_cast<const XE *>(x + (uint64_t)(VMODE == 2 ? w >> 8 : w) * stride);
        if constexpr (XC) xe[u] = M::ldB(p);
        else xe[u] = M::ldS(p);
        if constexpr (VMODE == 0) d[u] = FULL || u < left ? ldv(data + k + u) : vzero<DV>();
        if constexpr (VMODE == 1) d[u] = tab[FULL || u < left ? (uint32_t)__ldcs(codes + k + u) : 0u];
    }
#pragma unroll
    for (int u = 0; u < VB; u++) {
        if (FULL || u < left) {
            if constexpr (XC) vmul_acc<M>(ar[u % NC], ai[u % NC], d[u], xe[u]);
            else rmul_acc<M>(ar[u % NC], ai[u % NC], d[u], xe[u]);
        }
    }
}

// Sum of one row for one vector, with the vectors across the lanes: a group
// of VL lanes owns a row and lane v of it vector c, so one warp load gathers
// the VL vectors' entries of a nonzero as one contiguous piece.  The group's
// column words are loaded VB at a time, WPL per lane (one, or two where VL is 2
// or 3), a batch ahead of their use, and handed round by shuffles.  The loop is
// bound by its instruction count (issue slots 64% busy in the product of the L = 20
// Ising sector with 8 vectors), nearly all of it float-pair arithmetic: batches that every row of
// the warp fills run without predicates, addresses are one 32 x 32
// multiply-add, and lanes past the last vector (c clamped by the caller) load
// and compute like the rest.  Every lane of the warp calls it with its row's
// range (empty for none).  LONG: parts of a row take every split-th batch of it,
// and the whole sum is in part 0.  x: the vectors' base at vector c; stride: bytes
// per row of vectors (64 bits where they pass 4 GB).  VMODE: 0 one value per
// nonzero, 1 coded, 2 codes packed into the column words (tab: the 256 values).
template <class M, class DV, bool XC, class IT, int VMODE, int WPL, bool LONG, class ST>
__device__ __forceinline__ void vl_row_sum(const int32_t *__restrict__ indices, const DV *__restrict__ data,
                                           const uint8_t *__restrict__ codes, const DV *tab, const void *x,
                                           ST stride, int v, int lane0, int part, bool owns, int VL, int parts, IT k0, IT k1,
                                           typename M::S &sr, typename M::S &si)
{
    constexpr int NC = VCHAINS<M, LONG>;
    constexpr bool FLUSH = NC == 4;
    const int split = LONG ? parts : 1;
    int len = (int)(k1 - k0);
    const int most = __reduce_max_sync(0xffffffffu, len), step = split * VB;
    const int least = __reduce_min_sync(0xffffffffu, owns ? len : most);   // of the lanes that own a row
    const char *xb = reinterpret_cast<const char *>(x);
    const bool loads = v * WPL < VB;           // the lanes that fetch the words
    // this part's first batch; a lane without a row stays below `least` in a full batch
    if constexpr (LONG) {
        k0 += (IT)(part * VB);
        len -= part * VB;
    }
    uint32_t word[WPL];
    auto fetch = [&](int b) {
#pragma unroll
        for (int i = 0; i < WPL; i++) {
            const int k = b + v * WPL + i;
            word[i] = loads && k < len ? (uint32_t)__ldcs(indices + k0 + k) : 0u;
        }
    };
    typename M::S ar[NC], ai[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) ar[i] = ai[i] = M::zero();
    fetch(0);
    typename M::S tr = M::zero(), ti = M::zero();
    for (int b = 0, t = 1; b < most; b += step, t++) {
        uint32_t cur[WPL];
#pragma unroll
        for (int i = 0; i < WPL; i++) cur[i] = word[i];
        fetch(b + step);
        if (b + step <= least)
            vl_batch<M, DV, XC, IT, VMODE, WPL, true>(cur, lane0, data, codes, tab, xb, stride, k0 + b, VB, ar, ai);
        else
            vl_batch<M, DV, XC, IT, VMODE, WPL, false>(cur, lane0, data, codes, tab, xb, stride, k0 + b, len - b, ar, ai);
        if constexpr (FLUSH) {
            if (t % VFLUSH == 0) {
                tr = M::add(tr, M::add(M::add(ar[0], ar[2]), M::add(ar[1], ar[3])));
                ti = M::add(ti, M::add(M::add(ai[0], ai[2]), M::add(ai[1], ai[3])));
#pragma unroll
                for (int i = 0; i < NC; i++) ar[i] = ai[i] = M::zero();
            }
        }
    }
#pragma unroll
    for (int h = NC / 2; h > 0; h /= 2)
#pragma unroll
        for (int i = 0; i < h; i++) {
            ar[i] = M::merge(ar[i], ar[i + h]);
            ai[i] = M::merge(ai[i], ai[i + h]);
        }
    sr = FLUSH ? M::add(tr, ar[0]) : ar[0];
    si = FLUSH ? M::add(ti, ai[0]) : ai[0];
    if constexpr (LONG)
        for (int o = 1; o < split; o <<= 1) {
            const int from = (threadIdx.x & 31) + o * VL;
            sr = M::merge(sr, M::shfl(sr, from));
            si = M::merge(si, M::shfl(si, from));
        }
}

}  // namespace
