// CSR SpMV / SpMM without FP64 instructions per nonzero.
//
// y = a A x (overwrite) or y += a A x, the contract of parallel-sparse-tools'
// _matvec (docs/modules/parallel_sparse_tools/matvec/matvec_core.html:146-201
// in the reference), in two arithmetic forms (csrc/lp_modes.cuh):
//
//   * paired single (qs_csr_matvec_pairs): float64 / complex128 x and y, the
//     matrix values as float pairs (qs_split_pairs).  x is first scaled by
//     the power of two at or below its largest component and split into
//     pairs (two streaming passes over x), the products and row sums run in
//     FP32 instructions with 48-bit significands, and the scale is undone
//     exactly when the row result is converted to double;
//   * single precision (qs_csr_matvec with float32 / complex64 x and values):
//     FP32 products and row sums, float32 / complex64 y.
//
// One vector: row hand-out, lanes per row and entries in flight follow
// csrc/sparse.cu; after the butterfly reduction lanes 0 and 1 of a row group
// write the real and imaginary part of y.  Several vectors: the vectors
// across the lanes.
#include "qs_common.cuh"
#include "pairf.cuh"
#include "lp_lanes.cuh"
#include "lanczos.cuh"
#include "sell.cuh"

namespace {

template <class T> struct is_cx { static constexpr bool value = false; };
template <class S> struct is_cx<cx<S>> { static constexpr bool value = true; };

// output stores: YT double / float (real) or cdbl / cflt (complex)
template <class M> __device__ __forceinline__ void st_out(double *y, int64_t e, int, typename M::S v, int k, int ow)
{
    double r = M::to_d(v, k);
    if (!ow) r += y[e];
    y[e] = r;
}
template <class M> __device__ __forceinline__ void st_out(cdbl *y, int64_t e, int comp, typename M::S v, int k, int ow)
{
    double *p = reinterpret_cast<double *>(y + e) + comp;
    double r = M::to_d(v, k);
    if (!ow) r += *p;
    *p = r;
}
template <class M> __device__ __forceinline__ void st_out(float *y, int64_t e, int, typename M::S v, int, int ow)
{
    float r = M::hi(v);
    if (!ow) r += y[e];
    y[e] = r;
}
template <class M> __device__ __forceinline__ void st_out(cflt *y, int64_t e, int comp, typename M::S v, int, int ow)
{
    float *p = reinterpret_cast<float *>(y + e) + comp;
    float r = M::hi(v);
    if (!ow) r += *p;
    *p = r;
}

// Sum of one row over its group's G lanes (every lane of the group gets it).
// VM: 0 one value per nonzero; 1 coded: data holds a table of QS_CODE_TABLE
// values followed by one code byte per nonzero (pdtype QS_PF8 / QS_CPF8);
// 2 packed: indices holds col << 8 | code and data the table only (QS_PF8P /
// QS_CPF8P); 3 packed, one complex vector, the column words read four per
// 16-byte load (indices readable up to the next multiple of four words).
// tab: the table in shared memory.
template <class M, class DV, bool XC, class IT, int U, int VM>
__device__ __forceinline__ void row_sum(const int32_t *__restrict__ indices, const DV *__restrict__ data,
                                        const uint8_t *__restrict__ codes, const DV *s_tab,
                                        const void *__restrict__ xv, unsigned long long keep, IT k0, IT k1, int lane,
                                        int G, typename M::S &ar, typename M::S &ai)
{
    using S = typename M::S;
    using BE = typename M::BE;
    const BE *xc = reinterpret_cast<const BE *>(xv);
    const S *xr = reinterpret_cast<const S *>(xv);
    ar = ai = M::zero();
    if constexpr (VM == 3) {
        // the row's packed column words in 16-byte aligned groups of four,
        // group g of the row to lane g mod G
        for (IT c = (k0 & ~(IT)3) + 4 * lane; c < k1; c += (IT)(4 * G)) {
            const uint4 w4 = __ldcs(reinterpret_cast<const uint4 *>(indices + c));
            const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int h = 0; h < 4; h += 2) {
                BE bv[2];
#pragma unroll
                for (int i = 0; i < 2; i++)
                    bv[i] = (c + h + i >= k0 && c + h + i < k1) ? M::ldB(xc + (int32_t)(w[h + i] >> 8), keep)
                                                                : BE{M::zero(), M::zero()};
#pragma unroll
                for (int i = 0; i < 2; i++)
                    if (c + h + i >= k0 && c + h + i < k1) vmul_acc<M>(ar, ai, s_tab[w[h + i] & 255u], bv[i]);
            }
        }
    } else {
        for (IT k = k0 + lane; k < k1; k += (IT)(G * U)) {
            int32_t col[U];
            DV d[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const IT kk = k + (IT)(u * G);
                const bool in = kk < k1;
                if constexpr (VM == 2) {
                    const uint32_t w = in ? (uint32_t)__ldcs(indices + kk) : 0u;
                    col[u] = (int32_t)(w >> 8);
                    d[u] = in ? s_tab[w & 255u] : vzero<DV>();
                } else {
                    col[u] = in ? __ldcs(indices + kk) : 0;
                    if constexpr (VM == 1) d[u] = in ? s_tab[__ldcs(codes + kk)] : vzero<DV>();
                    else d[u] = in ? ldv(data + kk) : vzero<DV>();
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (k + (IT)(u * G) < k1) {
                    if constexpr (XC) vmul_acc<M>(ar, ai, d[u], M::ldB(xc + col[u], keep));
                    else rmul_acc<M>(ar, ai, d[u], M::ldS(xr + col[u]));
                }
            }
        }
    }
    for (int o = G >> 1; o > 0; o >>= 1) {
        ar = M::merge(ar, M::shfl_xor(ar, o));
        if constexpr (XC || is_cx<DV>::value) ai = M::merge(ai, M::shfl_xor(ai, o));
    }
}

// One vector (VM: see row_sum); the table is staged in shared memory.
template <class M, class DV, bool XC, class YT, class IT, int U, int VM>
__global__ void __launch_bounds__(256) spmv_lp_kernel(int64_t n, int lgG, const IT *__restrict__ indptr,
                                                      const int32_t *__restrict__ indices,
                                                      const DV *__restrict__ data, const void *__restrict__ xv,
                                                      YT *__restrict__ y, cdbl a, int overwrite,
                                                      const unsigned long long *__restrict__ xnorm)
{
    using S = typename M::S;
    constexpr bool COUT = XC || is_cx<DV>::value;
    __shared__ S s_a[2];
    __shared__ int s_k;
    if (threadIdx.x == 0) s_a[0] = M::from_d(a.x);
    if (threadIdx.x == 1) s_a[1] = M::from_d(a.y);
    if (threadIdx.x == 2) s_k = xnorm ? scale_exp(__longlong_as_double((long long)*xnorm)) : 0;
    constexpr bool CODED = VM != 0;
    __shared__ DV s_tab[CODED ? QS_CODE_TABLE : 1];
    const uint8_t *codes = nullptr;
    if constexpr (CODED) {
        for (int i = threadIdx.x; i < QS_CODE_TABLE; i += blockDim.x) s_tab[i] = ldv(data + i);
        codes = reinterpret_cast<const uint8_t *>(data + QS_CODE_TABLE);
    }
    __syncthreads();
    const cx<S> av{s_a[0], s_a[1]};
    const int k2 = s_k;
    const unsigned long long keep = l2_keep_policy();

    const int G = 1 << lgG;
    const int GPW = 32 >> lgG;
    const int lane = threadIdx.x & (G - 1);
    const int comp = lane & 1;
    const int gsub = (threadIdx.x & 31) >> lgG;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t rb = warp * GPW; rb < n; rb += nwarps * GPW) {
        const int64_t r = rb + gsub;
        const bool valid = r < n;
        const bool writer = valid && (COUT ? lane < 2 : lane == 0);
        const IT k0 = valid ? indptr[r] : (IT)0, k1 = valid ? indptr[r + 1] : (IT)0;
        S ar, ai;
        row_sum<M, DV, XC, IT, U, VM>(indices, data, codes, s_tab, xv, keep, k0, k1, lane, G, ar, ai);
        if (writer) {
            const S accr = M::fin(ar);
            if constexpr (COUT) {
                const S acci = M::fin(ai);
                const S v = comp ? M::add(M::mul(av.re, acci), M::mul(av.im, accr))
                                 : M::sub(M::mul(av.re, accr), M::mul(av.im, acci));
                st_out<M>(y, r, comp, v, k2, overwrite);
            } else {
                st_out<M>(y, r, 0, M::mul(av.re, accr), k2, overwrite);
            }
        }
    }
}

// The product of a Lanczos step with the rest of its row work: r = A q - b v
// and the block's share of Re <q, r> (csrc/lanczos.cu: the step; xs: q split
// into pairs at a fixed scale).  The same row sums as spmv_lp_kernel;
// the three FP64 instructions per component ride on rows that are otherwise
// bound by their gathers, and r is written once.
template <class DV, bool XC, int U, int VM>
__global__ void __launch_bounds__(256) spmv_lz_kernel(LzProduct p, int lgG)
{
    using M = ModePF;
    constexpr bool CODED = VM != 0;
    __shared__ DV s_tab[CODED ? QS_CODE_TABLE : 1];
    if (p.ctl->done) return;
    const DV *data = reinterpret_cast<const DV *>(p.data);
    if constexpr (CODED) {
        for (int i = threadIdx.x; i < QS_CODE_TABLE; i += blockDim.x) s_tab[i] = ldv(data + i);
        __syncthreads();
    }
    const int32_t *__restrict__ indptr = p.indptr;
    const unsigned long long keep = l2_keep_policy();
    const double bv = p.v ? *p.b : 0.0;
    const int G = 1 << lgG, GPW = 32 >> lgG, lane = threadIdx.x & (G - 1), comp = lane & 1;
    const int gsub = (threadIdx.x & 31) >> lgG;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    double dot = 0.0;
    for (int64_t rb = warp * GPW; rb < p.n; rb += nwarps * GPW) {
        const int64_t r = rb + gsub;
        const bool valid = r < p.n;
        const int32_t k0 = valid ? indptr[r] : 0, k1 = valid ? indptr[r + 1] : 0;
        pf ar, ai;
        row_sum<M, DV, XC, int32_t, U, VM>(p.indices, data, nullptr, s_tab, p.xs, keep, k0, k1, lane, G, ar, ai);
        if (valid && (XC ? lane < 2 : lane == 0)) {
            const int64_t e = XC ? 2 * r + comp : r;
            double rr = M::to_d(M::fin(XC && comp ? ai : ar), -p.xexp);
            if (p.v) rr = fma(-bv, __ldg(p.v + e), rr);
            p.r[e] = rr;
            dot = fma(__ldg(p.q + e), rr, dot);
        }
    }
    lz_block_finish(dot, p.partial, p.alpha, LZ_SUM, 0.0, 0, nullptr, p.ctl);
}

// Several vectors: the vectors across the lanes (vl_row_sum), VL lanes to a
// row, sweeps of VL vectors.  With the vectors on the accumulators of one lane
// instead, a warp's load of one vector touches 32 lines for 32 nonzeros and is
// bound by the L1 tag rate.  Measured (whole product, x split included), the
// Ising chain L = 22 at k != 0 (191 k rows, 4.4 M complex nonzeros): 8 vectors
// 194 us then, 120 us now; 5 vectors 112 / 87 us; J1-J2 L = 28 (361 k rows,
// 10.7 M real nonzeros): 8 vectors 401 / 191 us, 2 vectors 98 / 69 us.  Complex
// pairs run at three blocks per SM (four spill: 129 us), the rest at four.
// LONG: as vl_row_sum, with sweeps of the vectors for gridDim.y.
template <class M, class DV, bool XC, class YT, class IT, int VM, int WPL, class ST, bool LONG>
__global__ void __launch_bounds__(256, std::is_same<DV, cpf>::value ? 3 : 4)
spmm_vl_kernel(int64_t n, const IT *__restrict__ indptr, const int32_t *__restrict__ indices,
               const DV *__restrict__ data, const void *__restrict__ xv, YT *__restrict__ y, int64_t nvec, int VL,
               int parts, cdbl a, int overwrite, const unsigned long long *__restrict__ xnorm)
{
    using S = typename M::S;
    using XE = typename std::conditional<XC, typename M::BE, S>::type;
    constexpr bool COUT = XC || is_cx<DV>::value;
    __shared__ S s_a[2];
    __shared__ int s_k;
    if (threadIdx.x == 0) s_a[0] = M::from_d(a.x);
    if (threadIdx.x == 1) s_a[1] = M::from_d(a.y);
    if (threadIdx.x == 2) s_k = xnorm ? scale_exp(__longlong_as_double((long long)*xnorm)) : 0;
    constexpr bool CODED = VM != 0;
    __shared__ DV s_tab[CODED ? QS_CODE_TABLE : 1];
    const uint8_t *codes = nullptr;
    if constexpr (CODED) {
        for (int i = threadIdx.x; i < QS_CODE_TABLE; i += blockDim.x) s_tab[i] = ldv(data + i);
        codes = reinterpret_cast<const uint8_t *>(data + QS_CODE_TABLE);
    }
    __syncthreads();
    const cx<S> av{s_a[0], s_a[1]};
    const int k2 = s_k;
    const int split = LONG ? parts : 1;
    const int64_t first = LONG ? (int64_t)blockIdx.y * VL : 0, sweep = LONG ? (int64_t)gridDim.y * VL : VL;
    // the short form written out: with vl_place the compiler's schedule of the whole
    // loop is up to 5% slower (70 k rows of 24, 8 vectors, 41.3 against 39.4 us)
    VlPlace at;
    if constexpr (LONG) at = vl_place(VL, split);
    else {
        at.rows = 32 / VL;
        at.grp = (threadIdx.x & 31) / VL;
        at.lane0 = at.grp * VL;
        at.v = (threadIdx.x & 31) - at.lane0;
        at.part = 0;
    }
    const int v = at.v;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t rb = warp * at.rows; rb < n; rb += nwarps * at.rows) {
        const int64_t r = rb + at.grp;
        const bool valid = r < n && at.grp < at.rows;
        const IT k0 = valid ? indptr[r] : (IT)0, k1 = valid ? indptr[r + 1] : (IT)0;
        for (int64_t c0 = first; c0 < nvec; c0 += sweep) {
            const int64_t c = c0 + v < nvec ? c0 + v : nvec - 1;
            const bool act = valid && at.part == 0 && c0 + v < nvec;
            S ar = M::zero(), ai = M::zero();
            vl_row_sum<M, DV, XC, IT, VM, WPL, LONG>(indices, data, codes, s_tab,
                                                     reinterpret_cast<const XE *>(xv) + c, (ST)(nvec * sizeof(XE)),
                                                     v, at.lane0, at.part, at.grp < at.rows, VL, split, k0, k1, ar, ai);
            if (act) {
                const int64_t e = r * nvec + c;
                const S accr = M::fin(ar);
                if constexpr (COUT) {
                    const S acci = M::fin(ai);
                    st_out<M>(y, e, 0, M::sub(M::mul(av.re, accr), M::mul(av.im, acci)), k2, overwrite);
                    st_out<M>(y, e, 1, M::add(M::mul(av.re, acci), M::mul(av.im, accr)), k2, overwrite);
                } else {
                    st_out<M>(y, e, 0, M::mul(av.re, accr), k2, overwrite);
                }
            }
        }
    }
}

// The power of two at the largest |component| of a double array, as the high
// word of a double in *norm (scale_exp reads its exponent only).  Integer
// compares of the high words: an FP64 maximum is two FP64-pipe instructions.
// NaN counts as nothing, as in an FP64 maximum.
__global__ void __launch_bounds__(256) xnorm_kernel(int64_t count, const double *__restrict__ x,
                                                    unsigned long long *norm)
{
    uint32_t m = 0;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += step) {
        const double v = __ldg(x + i);
        uint32_t h = (uint32_t)__double2hiint(v) & 0x7fffffffu;
        if (h >= 0x7ff00000u && (h > 0x7ff00000u || __double2loint(v) != 0)) h = 0u;
        m = h > m ? h : m;
    }
    // one atomic per block: all of them meet at one address
    __shared__ uint32_t s_m[8];
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 8) {
        m = __reduce_max_sync(0xffu, s_m[threadIdx.x]);
        if (threadIdx.x == 0 && m) atomicMax(norm, (unsigned long long)m << 32);
    }
}

// xs[i] = pair(x[i] 2^-k), k from *norm
__global__ void __launch_bounds__(256) xsplit_kernel(int64_t count, const double *__restrict__ x,
                                                     float2 *__restrict__ xs,
                                                     const unsigned long long *__restrict__ norm)
{
    const int k = scale_exp(__longlong_as_double((long long)*norm));
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += step) {
        const pf v = pair_rn_scaled(__ldcs(x + i), k);
        xs[i] = make_float2(v.h, v.l);
    }
}

struct SpmvArgs {
    int64_t n, nnz;
    const void *indptr;
    int idx64;
    const int32_t *indices;
    const void *data;
    const void *x;
    void *y;
    int64_t nvec;
    cdbl a;
    int overwrite;
    const unsigned long long *xnorm;
    int G, U;
    cudaStream_t st;
};

static int grid_rows(int64_t n, int G)
{
    int64_t gpb = 256 / G;
    int64_t b = (n + gpb - 1) / gpb;
    int64_t cap = (int64_t)qs_num_sms() * 16;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

template <class M, class DV, bool XC, class YT, class IT, int U, int VM>
int spmv_go(const SpmvArgs &a)
{
    int lg = 0;
    while ((1 << lg) < a.G) lg++;
    // persistent grid (grid-stride kernel): one wave of resident blocks
    static int resident = 0;
    auto k = spmv_lp_kernel<M, DV, XC, YT, IT, U, VM>;
    const int blocks = qs_persistent_grid(k, 256, grid_rows(a.n, a.G), resident);
    k<<<blocks, 256, 0, a.st>>>(a.n, lg, (const IT *)a.indptr, a.indices, (const DV *)a.data, a.x, (YT *)a.y, a.a,
                                a.overwrite, a.xnorm);
    QS_CHECK(cudaGetLastError());
    return QS_OK;
}

template <class M, class DV, bool XC, class YT, class IT, int VM, int WPL, class ST, bool LONG>
int spmm_run(const SpmvArgs &a, int VL, int split, int64_t lanes)
{
    static int resident = 0;
    auto k = spmm_vl_kernel<M, DV, XC, YT, IT, VM, WPL, ST, LONG>;
    const int64_t rows = 8 * (32 / (VL * split));       // per block and sweep
    // with few rows the sweeps go to blocks of their own, too
    int64_t apart = LONG ? lanes / (a.n * VL * split) : 1;
    if (apart > 65535) apart = 65535;
    if (apart > (a.nvec + VL - 1) / VL) apart = (a.nvec + VL - 1) / VL;
    const dim3 grid(qs_persistent_grid(k, 256, (a.n + rows - 1) / rows, resident), (unsigned)(apart < 1 ? 1 : apart));
    k<<<grid, 256, 0, a.st>>>(a.n, (const IT *)a.indptr, a.indices, (const DV *)a.data, a.x, (YT *)a.y, a.nvec, VL,
                              split, a.a, a.overwrite, a.xnorm);
    QS_CHECK(cudaGetLastError());
    return QS_OK;
}

template <class M, class DV, bool XC, class YT, class IT, int VM, int WPL, class ST = uint32_t>
int spmm_go(const SpmvArgs &a)
{
    // FP32 arithmetic leaves more of the latency to hide than float pairs do
    const int64_t lanes = std::is_same<M, ModeF32>::value ? 130000 : 100000;
    const int VL = vl_lanes(a.nvec), split = vl_split(a.n, a.nnz, VL, lanes);
    if constexpr (sizeof(ST) == 4) {
        if (!vl_long<M>(a.n, a.nnz, split)) return spmm_run<M, DV, XC, YT, IT, VM, WPL, ST, false>(a, VL, 1, lanes);
    }
    return spmm_run<M, DV, XC, YT, IT, VM, WPL, ST, true>(a, VL, split, lanes);
}

template <class M, class DV, bool XC, class YT, class IT, int VM>
int spmv_nb(const SpmvArgs &a)
{
    if constexpr (VM == 3) {
        if (a.nvec != 1 || !XC) return QS_ERR_ARG;
        return spmv_go<M, DV, XC, YT, IT, 1, 3>(a);
    } else {
        if (a.nvec == 1) {
            if constexpr (sizeof(IT) == 4) {
                if (a.U >= 4) return spmv_go<M, DV, XC, YT, IT, 4, VM>(a);
                if (a.U >= 2) return spmv_go<M, DV, XC, YT, IT, 2, VM>(a);
            }
            return spmv_go<M, DV, XC, YT, IT, 1, VM>(a);
        }
        // a row of the vectors beyond 4 GB
        if (a.nvec > (int64_t)(0xffffffffu / (XC ? sizeof(typename M::BE) : sizeof(typename M::S))))
            return spmm_go<M, DV, XC, YT, IT, VM, 1, uint64_t>(a);
        if (a.nvec <= 3) return spmm_go<M, DV, XC, YT, IT, VM, 2>(a);
        return spmm_go<M, DV, XC, YT, IT, VM, 1>(a);
    }
}

// coded and packed values: int32 column indices only
template <class M, class DV, bool XC, class YT, int VM = 0>
int spmv_idx(const SpmvArgs &a)
{
    if constexpr (VM != 0) {
        if (a.idx64) return QS_ERR_ARG;
        return spmv_nb<M, DV, XC, YT, int32_t, VM>(a);
    } else {
        if (a.idx64) return spmv_nb<M, DV, XC, YT, int64_t, 0>(a);
        return spmv_nb<M, DV, XC, YT, int32_t, 0>(a);
    }
}

}  // namespace

// float32 / complex64 operands (called by qs_csr_matvec): 0 when handled,
// QS_ERR_UNSUPPORTED for type pairs left to the double kernels.
int spmv_lp_single(int64_t n, int64_t nnz, const void *indptr, int idx64, const int32_t *indices, const void *data, int dtype,
                   const void *x, int xtype, void *y, int64_t nvec, cdbl a, int overwrite, int G, int U,
                   cudaStream_t st)
{
    SpmvArgs s{n, nnz, indptr, idx64, indices, data, x, y, nvec, a, overwrite, nullptr, G, U, st};
    if (xtype == QS_F32 && dtype == QS_F32) return spmv_idx<ModeF32, float, false, float>(s);
    if (xtype == QS_C64 && dtype == QS_F32) return spmv_idx<ModeF32, float, true, cflt>(s);
    if (xtype == QS_C64 && dtype == QS_C64) return spmv_idx<ModeF32, cx<float>, true, cflt>(s);
    return QS_ERR_UNSUPPORTED;
}

namespace {
template <class DV, bool XC, int U, int VM>
int lz_go(const LzProduct &p, int G, cudaStream_t st)
{
    int lg = 0;
    while ((1 << lg) < G) lg++;
    static int resident = 0;
    auto k = spmv_lz_kernel<DV, XC, U, VM>;
    k<<<qs_persistent_grid(k, 256, grid_rows(p.n, G), resident), 256, 0, st>>>(p, lg);
    QS_CHECK(cudaGetLastError());
    return QS_OK;
}
template <class DV, bool XC, int VM>
int lz_u(const LzProduct &p, int G, int U, cudaStream_t st)
{
    if (U >= 4) return lz_go<DV, XC, 4, VM>(p, G, st);
    if (U >= 2) return lz_go<DV, XC, 2, VM>(p, G, st);
    return lz_go<DV, XC, 1, VM>(p, G, st);
}
}  // namespace

// The fused product of a Lanczos step: plain pairs or packed codes (int32
// row pointers), launch shape `group` as for qs_csr_matvec_pairs.
int spmv_lanczos(const LzProduct &p, int pdtype, int cplx, int group, cudaStream_t st)
{
    if (sell_type(pdtype)) return sell_lanczos(p, pdtype, cplx, st);
    int G = group > 0 ? (group & 0xff) : 2, U = group > 0 ? ((group >> 8) & 0xff) : 1;
    if (G != 2 && G != 4 && G != 8 && G != 16 && G != 32) return QS_ERR_ARG;
    const bool v4 = group > 0 && ((group >> 20) & 7) == 6;
    switch (pdtype) {
    case QS_PF: return cplx ? lz_u<pf, true, 0>(p, G, U, st) : lz_u<pf, false, 0>(p, G, U, st);
    case QS_CPF: return cplx ? lz_u<cpf, true, 0>(p, G, U, st) : QS_ERR_ARG;
    case QS_PF8P:
        if (v4) return cplx ? lz_go<pf, true, 1, 3>(p, G, st) : QS_ERR_ARG;
        return cplx ? lz_u<pf, true, 2>(p, G, U, st) : lz_u<pf, false, 2>(p, G, U, st);
    case QS_CPF8P:
        if (!cplx) return QS_ERR_ARG;
        return v4 ? lz_go<cpf, true, 1, 3>(p, G, st) : lz_u<cpf, true, 2>(p, G, U, st);
    default: return QS_ERR_ARG;
    }
}

// y = a A x (overwrite) or y += a A x with float64 / complex128 x and y and
// the matrix values as float pairs (pdtype QS_PF from float64 values,
// QS_CPF from complex128 values; a complex matrix needs complex x), or as
// one code byte per nonzero into a table of such pairs (QS_PF8 / QS_CPF8:
// QS_CODE_TABLE pairs, then nnz uint8 codes; int32 indices), or with the
// code packed into the low 8 bits of each column word (QS_PF8P / QS_CPF8P:
// indices holds col << 8 | code, col < 2^23; pdata the table only), or such
// words in slices of 32 rows (QS_PF8S / QS_CPF8S, one vector: csrc/sell.cu;
// indptr holds the slice pointers, int64).
// xs: scratch of n*nvec*(8 or 16) bytes for the split x; norm: 8 bytes of
// device scratch.  group as for qs_csr_matvec.
extern "C" int qs_csr_matvec_pairs(int64_t n, int64_t nnz, const void *indptr, int idx64, const int32_t *indices,
                                   const void *pdata, int pdtype, const void *x, int xtype, void *y, int64_t nvec,
                                   double a_re, double a_im, int overwrite, int group, void *xs, void *norm,
                                   void *stream)
{
    if (n < 0 || nvec < 1 || (n > 0 && (!indptr || !x || !y || !xs || !norm))) return QS_ERR_ARG;
    if (n == 0) return QS_OK;
    const bool xc = xtype == QS_C128;
    if (!xc && xtype != QS_F64) return QS_ERR_ARG;
    const bool cvals = pdtype == QS_CPF || pdtype == QS_CPF8 || pdtype == QS_CPF8P || pdtype == QS_CPF8S;
    if (!xc && (a_im != 0.0 || cvals)) return QS_ERR_ARG;
    if (pdtype != QS_PF && pdtype != QS_CPF && pdtype != QS_PF8 && pdtype != QS_CPF8 && pdtype != QS_PF8P &&
        pdtype != QS_CPF8P && !sell_type(pdtype))
        return QS_ERR_ARG;
    if (sell_type(pdtype) && nvec != 1) return QS_ERR_ARG;
    if (pdtype != QS_PF && pdtype != QS_CPF && idx64) return QS_ERR_ARG;
    int G = group > 0 ? (group & 0xff) : 2;
    int U = group > 0 ? ((group >> 8) & 0xff) : 1;
    if (U < 1) U = 1;
    if (G != 2 && G != 4 && G != 8 && G != 16 && G != 32) return QS_ERR_ARG;
    if (U != 1 && U != 2 && U != 4) return QS_ERR_ARG;
    (void)nnz;
    cudaStream_t st = qs_stream(stream);
    unsigned long long *nrm = reinterpret_cast<unsigned long long *>(norm);
    const int64_t count = n * nvec * (xc ? 2 : 1);
    QS_CHECK(cudaMemsetAsync(nrm, 0, sizeof(unsigned long long), st));
    int64_t b = (count + 255) / 256, cap = (int64_t)qs_num_sms() * 8;
    const int blocks = (int)(b > cap ? cap : b), nblk = (int)(b > cap / 2 ? cap / 2 : b);
    xnorm_kernel<<<nblk, 256, 0, st>>>(count, (const double *)x, nrm);
    xsplit_kernel<<<blocks, 256, 0, st>>>(count, (const double *)x, (float2 *)xs, nrm);
    QS_CHECK(cudaGetLastError());
    if (sell_type(pdtype))
        return sell_spmv(n, (const int64_t *)indptr, indices, pdata, pdtype, xs, xc, y, cdbl{a_re, a_im}, overwrite, nrm,
                         st);
    SpmvArgs s{n, nnz, indptr, idx64, indices, pdata, xs, y, nvec, cdbl{a_re, a_im}, overwrite, nrm, G, U, st};
    if (pdtype == QS_PF8) return xc ? spmv_idx<ModePF, pf, true, cdbl, 1>(s) : spmv_idx<ModePF, pf, false, double, 1>(s);
    if (pdtype == QS_CPF8) return spmv_idx<ModePF, cpf, true, cdbl, 1>(s);
    const bool v4 = ((group >> 20) & 7) == 6 && group > 0;
    if (v4 && !(xc && nvec == 1 && (pdtype == QS_PF8P || pdtype == QS_CPF8P))) return QS_ERR_ARG;
    if (pdtype == QS_PF8P) {
        if (v4) return spmv_idx<ModePF, pf, true, cdbl, 3>(s);
        return xc ? spmv_idx<ModePF, pf, true, cdbl, 2>(s) : spmv_idx<ModePF, pf, false, double, 2>(s);
    }
    if (pdtype == QS_CPF8P) return v4 ? spmv_idx<ModePF, cpf, true, cdbl, 3>(s) : spmv_idx<ModePF, cpf, true, cdbl, 2>(s);
    if (!xc) return spmv_idx<ModePF, pf, false, double>(s);
    if (pdtype == QS_PF) return spmv_idx<ModePF, pf, true, cdbl>(s);
    return spmv_idx<ModePF, cpf, true, cdbl>(s);
}
