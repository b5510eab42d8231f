// Single-vector products on a sliced operand.
//
// The row hand-out kernels are bound by L1: a warp's gather of 32 nonzeros
// touches one 128-byte line per lane or nearly so (0.63 lines per nonzero in the
// J1-J2 sectors), and each line is a tag lookup.  Neighbouring rows do have
// neighbouring columns: the 32 rows of a slice touch only 0.29 distinct lines
// per nonzero, but at different places of their rows.
//
// Here a warp takes a slice of 32 rows, one row per lane, and walks its slots:
// in slot k every lane gathers one nonzero of its row.  The order of a row's
// nonzeros over the slots is free, so it is chosen for all 32 rows together
// (sell_fill_kernel): nonzeros of different rows that read the same line go
// into the same slot where they can.  Lines per nonzero, row hand-out -> sliced:
// J1-J2 L = 28 0.63 -> 0.34, XXZ L = 26 -> 0.30, Ising L = 18 -> 0.31 (distinct
// lines of a slice, the least there could be: 0.29, 0.26, 0.25).
// Measured, the best row hand-out shape -> here: a Taylor term of J1-J2 L = 32
// (4.7 M rows, 159 M nonzeros) 524 -> 380 us, L = 30 143 -> 110, L = 28 50 -> 40;
// the product of a complex vector, its split into pairs included, 506 -> 383,
// 140 -> 112 and 50 -> 43 us, Ising L = 22 31 -> 29, XXZ L = 26 (rows of 5 to 27)
// 26 -> 25.  Re-ordering takes 4.9 ms at 159 M nonzeros, once per operator.
// Bound by issue slots (66%) and L1 (65%) about alike.  DRAM traffic of a term at
// L = 32, where the term vectors, F and the words exceed L2 together: 1.98 -> 1.04
// GB, 1.02 times what the padded words and the vectors once come to.
//
// The layout is of the sliced ELLPACK family (A. Monakov, A. Lokhmotov and A.
// Avetisyan, HiPEAC 2010; SELL-C-sigma, M. Kreutzer et al., SIAM J. Sci. Comput. 36
// (2014) C401-C423); the order of a slice's nonzeros over its slots is this file's.
//
// Words: col << 8 | code as in the packed form, PAD where a row has no nonzero
// in the slot; slots in groups of four, a group as 32 x 16 bytes, so that a
// lane loads four of its words at once.  sptr[s]: groups before slice s.
#include "sell.cuh"
#include "lp_lanes.cuh"

namespace {

constexpr uint32_t PAD = 0xffffffffu;      // column 2^24 - 1: packed columns are below 2^23
constexpr int MAX_SLOTS = 128;             // slots whose free rows a warp keeps in registers

// groups of four slots of each slice
__global__ void __launch_bounds__(256) sell_count_kernel(int64_t n, const int32_t *__restrict__ indptr,
                                                         int64_t *__restrict__ groups, int *__restrict__ most)
{
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int len = r < n ? indptr[r + 1] - indptr[r] : 0;
    const int top = __reduce_max_sync(0xffffffffu, len);
    if ((threadIdx.x & 31) == 0 && r < n) {
        groups[r >> 5] = (top + 3) / 4;
        atomicMax(most, top);
    }
}

// One warp per slice.  The rows are merged by line (their words ascend); the
// rows that have a word in the lowest line left form a group, which goes to the
// slot with the most of them still free, the fullest of those, then the rest of
// the group again.  A row meets every slot at most once, so it always has a
// free one.  Lane i holds the free rows of the slots i, i + 32, ...
__global__ void __launch_bounds__(256) sell_fill_kernel(int64_t n, const int32_t *__restrict__ indptr,
                                                        const int32_t *__restrict__ words,
                                                        const int64_t *__restrict__ sptr, uint32_t *__restrict__ out)
{
    constexpr int Q = MAX_SLOTS / 32;
    const int64_t slices = (n + 31) / 32, s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (s >= slices) return;
    const int lane = threadIdx.x & 31;
    const int64_t r = s * 32 + lane;
    int k = r < n ? indptr[r] : 0;
    const int k1 = r < n ? indptr[r + 1] : 0;
    const int64_t base = sptr[s] * 128;
    const int slots = (int)(sptr[s + 1] - sptr[s]) * 4;
    uint32_t free_[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) free_[q] = lane + 32 * q < slots ? 0xffffffffu : 0u;
    uint32_t w = k < k1 ? (uint32_t)__ldg(words + k) : PAD;
    uint32_t after = k + 1 < k1 ? (uint32_t)__ldg(words + k + 1) : PAD;
    for (;;) {
        const uint32_t line = __reduce_min_sync(0xffffffffu, w >> 11);      // 8 columns of 16 bytes
        if (line == PAD >> 11) break;
        uint32_t g = __ballot_sync(0xffffffffu, w >> 11 == line);
        while (g) {
            uint32_t best = 0;
#pragma unroll
            for (int q = 0; q < Q; q++) {
                if (32 * q >= slots) break;
                const uint32_t fit = __popc(free_[q] & g);
                const uint32_t score = fit << 13 | (32u - __popc(free_[q])) << 7 | (uint32_t)(127 - (lane + 32 * q));
                if (fit && score > best) best = score;
            }
            best = __reduce_max_sync(0xffffffffu, best);
            if (!best) return;                                              // cannot happen
            const int slot = 127 - (int)(best & 127u), owner = slot & 31;
            uint32_t take = 0;
#pragma unroll
            for (int q = 0; q < Q; q++)
                if (slot >> 5 == q) {
                    take = g & __shfl_sync(0xffffffffu, free_[q], owner);
                    if (lane == owner) free_[q] &= ~take;
                }
            g &= ~take;
            if (take >> lane & 1u) {
                out[base + (slot >> 2) * 128 + lane * 4 + (slot & 3)] = w;
                k++;
                w = after;
                after = k + 1 < k1 ? (uint32_t)__ldg(words + k + 1) : PAD;
            }
        }
    }
}

// Four slots: the lane's words w.  FULL: no lane has a PAD among them (most
// groups), so nothing is predicated; otherwise a PAD gathers column 0 and its
// product is skipped.
template <class DV, bool XC, bool FULL>
__device__ __forceinline__ void sell_group(const uint32_t (&w)[4], const DV *tab, const void *__restrict__ xv,
                                           unsigned long long keep, pf (&ar)[2], pf (&ai)[2])
{
    using M = ModePF;
    using XE = typename std::conditional<XC, cpf, pf>::type;
    XE xe[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const XE *x = reinterpret_cast<const XE *>(xv) + (FULL || w[u] != PAD ? w[u] >> 8 : 0u);
        if constexpr (XC) xe[u] = M::ldB(x, keep);
        else xe[u] = M::ldS(x);
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
        if (FULL || w[u] != PAD) {
            const DV d = tab[w[u] & 255u];
            if constexpr (XC) vmul_acc<M>(ar[u & 1], ai[u & 1], d, xe[u]);
            else rmul_acc<M>(ar[u & 1], ai[u & 1], d, xe[u]);
        }
}

// Sum of this lane's row of slice s, by the whole warp.  Even and odd slots on
// accumulators of their own, as two lanes of a row hand-out.
template <class DV, bool XC>
__device__ __forceinline__ void sell_row_sum(const int64_t *__restrict__ sptr, const int32_t *__restrict__ words,
                                             const DV *tab, const void *__restrict__ xv, unsigned long long keep,
                                             int64_t s, int lane, pf &sr, pf &si)
{
    using M = ModePF;
    const int64_t g0 = __ldg(sptr + s);
    const int groups = (int)(__ldg(sptr + s + 1) - g0);
    const uint4 *p = reinterpret_cast<const uint4 *>(words) + g0 * 32 + lane;
    pf ar[2] = {M::zero(), M::zero()}, ai[2] = {M::zero(), M::zero()};
    uint4 next = groups ? __ldcs(p) : make_uint4(PAD, PAD, PAD, PAD);
    for (int g = 0; g < groups; g++) {
        const uint32_t w[4] = {next.x, next.y, next.z, next.w};
        if (g + 1 < groups) next = __ldcs(p + (g + 1) * 32);
        const uint32_t top = max(max(w[0], w[1]), max(w[2], w[3]));
        if (__all_sync(0xffffffffu, top != PAD)) sell_group<DV, XC, true>(w, tab, xv, keep, ar, ai);
        else sell_group<DV, XC, false>(w, tab, xv, keep, ar, ai);
    }
    sr = M::merge(ar[0], ar[1]);
    si = M::merge(ai[0], ai[1]);
}

template <class DV>
__device__ __forceinline__ void sell_table(DV *s_tab, const void *data)
{
    for (int i = threadIdx.x; i < QS_CODE_TABLE; i += blockDim.x) s_tab[i] = ldv(reinterpret_cast<const DV *>(data) + i);
    __syncthreads();
}

// 64 registers a thread: 32 warps on an SM
constexpr int ST = 512, SOCC = 2;

template <class DV, bool XC>
__global__ void __launch_bounds__(ST, SOCC) sell_spmv_kernel(int64_t n, const int64_t *__restrict__ sptr,
                                                          const int32_t *__restrict__ words,
                                                          const void *__restrict__ data, const void *__restrict__ xv,
                                                          double *__restrict__ y, cdbl a, int overwrite,
                                                          const unsigned long long *__restrict__ xnorm)
{
    using M = ModePF;
    __shared__ DV s_tab[QS_CODE_TABLE];
    sell_table(s_tab, data);
    const unsigned long long keep = l2_keep_policy();
    const pf a_re = pair_rn_scaled(a.x, 0), a_im = pair_rn_scaled(a.y, 0);
    const int k2 = scale_exp(__longlong_as_double((long long)*xnorm)), lane = threadIdx.x & 31;
    const int64_t slices = (n + 31) / 32, nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < slices; s += nwarps) {
        pf sr, si;
        sell_row_sum<DV, XC>(sptr, words, s_tab, xv, keep, s, lane, sr, si);
        const int64_t r = s * 32 + lane;
        if (r >= n) continue;
        const pf accr = M::fin(sr);
        if constexpr (XC) {
            const pf acci = M::fin(si);
            double re = M::to_d(M::sub(M::mul(a_re, accr), M::mul(a_im, acci)), k2);
            double im = M::to_d(M::add(M::mul(a_re, acci), M::mul(a_im, accr)), k2);
            double2 *p = reinterpret_cast<double2 *>(y) + r;
            if (!overwrite) {
                const double2 o = *p;
                re += o.x;
                im += o.y;
            }
            *p = make_double2(re, im);
        } else {
            double re = M::to_d(M::mul(a_re, accr), k2);
            if (!overwrite) re += y[r];
            y[r] = re;
        }
    }
}

// The product of a Lanczos step (spmv_lz_kernel in csrc/spmv_lp.cu)
template <class DV, bool XC>
__global__ void __launch_bounds__(ST, SOCC) sell_lz_kernel(LzProduct p, const int64_t *__restrict__ sptr)
{
    using M = ModePF;
    __shared__ DV s_tab[QS_CODE_TABLE];
    if (p.ctl->done) return;
    sell_table(s_tab, p.data);
    const unsigned long long keep = l2_keep_policy();
    const double bv = p.v ? *p.b : 0.0;
    const int lane = threadIdx.x & 31;
    const int64_t slices = (p.n + 31) / 32, nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    double dot = 0.0;
    for (int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < slices; s += nwarps) {
        pf sr, si;
        sell_row_sum<DV, XC>(sptr, p.indices, s_tab, p.xs, keep, s, lane, sr, si);
        const int64_t r = s * 32 + lane;
        if (r >= p.n) continue;
        double re = M::to_d(M::fin(sr), -p.xexp);
        if constexpr (XC) {
            double im = M::to_d(M::fin(si), -p.xexp);
            if (p.v) {
                const double2 v = __ldg(reinterpret_cast<const double2 *>(p.v) + r);
                re = fma(-bv, v.x, re);
                im = fma(-bv, v.y, im);
            }
            const double2 q = __ldg(reinterpret_cast<const double2 *>(p.q) + r);
            reinterpret_cast<double2 *>(p.r)[r] = make_double2(re, im);
            dot = fma(q.x, re, dot);
            dot = fma(q.y, im, dot);
        } else {
            if (p.v) re = fma(-bv, __ldg(p.v + r), re);
            p.r[r] = re;
            dot = fma(__ldg(p.q + r), re, dot);
        }
    }
    lz_block_finish(dot, p.partial, p.alpha, LZ_SUM, 0.0, 0, nullptr, p.ctl);
}

// Running maximum over a warp's rows of |z|^2 formed in FP64.  The FP64
// instructions run only where the FP32 value says that some lane may pass what
// the warp has seen (an FP32 square is within a few 2^-23 of the FP64 one, the
// margin 2^-18): the maximum is the same to the bit, at about log of the number
// of slices instead of every slice.  Squares below the normal float range have
// no such bound and count as nothing seen, so that what follows passes; against
// a larger one, whose margin is 2^-144 or more, they cannot win.  NaN counts as
// nothing, as in fmax.
struct MaxSquare {
    double best = 0.0;
    uint32_t seen = 0u;      // bits of the largest FP32 value of the warp, less the margin
    __device__ __forceinline__ bool passes(float a, float b)
    {
        const float q = __fmaf_rn(a, a, __fmul_rn(b, b));
        const uint32_t top = __reduce_max_sync(0xffffffffu, q == q ? __float_as_uint(q) : 0u);
        if (top < seen) return false;
        seen = top < 0x00800000u    ? 0u
               : top >= 0x7f800000u ? top
                                    : __float_as_uint(__fmul_rn(__uint_as_float(top), 1.0f - 0x1p-18f));
        return true;
    }
    __device__ __forceinline__ void take(double a, double b) { best = fmax(best, __dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b))); }
};

// One Taylor term (the recurrence and the stopping test of csrc/expm_lp.cu,
// one vector), one row per lane.
template <class DV>
__global__ void __launch_bounds__(ST, SOCC) taylor_sell_kernel(int64_t n, const int64_t *__restrict__ sptr,
                                                            const int32_t *__restrict__ words,
                                                            const void *__restrict__ data,
                                                            const cpf *__restrict__ Bin, cpf *__restrict__ Bout,
                                                            cdbl *__restrict__ F, cdbl mu, const cdbl *__restrict__ coeff,
                                                            int j, double tol, ExpmCtl *ctl)
{
    using M = ModePF;
    __shared__ DV s_tab[QS_CODE_TABLE];
    if (*((volatile int *)&ctl->done)) return;
    const int bexp = *((volatile int *)&ctl->bexp);
    sell_table(s_tab, data);
    const unsigned long long keep = l2_keep_policy();
    const double s_inv = pow2(-bexp);
    const cdbl c = coeff[j];
    const pf cf_re = pair_rn_scaled(c.x, 0), cf_im = pair_rn_scaled(c.y, 0);
    const pf mu_re = pair_rn_scaled(mu.x, 0), mu_im = pair_rn_scaled(mu.y, 0);
    const pf cm_re = M::sub(M::mul(cf_re, mu_re), M::mul(cf_im, mu_im));
    const pf cm_im = M::add(M::mul(cf_re, mu_im), M::mul(cf_im, mu_re));
    const int lane = threadIdx.x & 31;
    const int64_t slices = (n + 31) / 32, nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    MaxSquare mb, mf;
    for (int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < slices; s += nwarps) {
        pf sr, si;
        sell_row_sum<DV, true>(sptr, words, s_tab, Bin, keep, s, lane, sr, si);
        const int64_t r = s * 32 + lane;
        const bool in = r < n;
        cpf bo{M::zero(), M::zero()};
        double2 f = make_double2(0.0, 0.0);
        if (in) {
            bo = M::ldB(Bin + r, keep);
            f = __ldcs(reinterpret_cast<const double2 *>(F + r));
        }
        // new term = cf (A B) - (cf mu) B
        const pf accr = M::fin(sr), acci = M::fin(si);
        cpf b;
        b.re = M::sub(M::sub(M::mul(cf_re, accr), M::mul(cf_im, acci)),
                      M::sub(M::mul(cm_re, bo.re), M::mul(cm_im, bo.im)));
        b.im = M::sub(M::add(M::mul(cf_re, acci), M::mul(cf_im, accr)),
                      M::add(M::mul(cm_re, bo.im), M::mul(cm_im, bo.re)));
        f.x = M::add_to(f.x, b.re, bexp);
        f.y = M::add_to(f.y, b.im, bexp);
        if (in) {
            M::st(Bout + r, b);
            __stcs(reinterpret_cast<double2 *>(F + r), f);
        } else {
            b = cpf{M::zero(), M::zero()};
            f = make_double2(0.0, 0.0);
        }
        if (mb.passes(b.re.h, b.im.h)) mb.take(M::to_d(b.re, 0), M::to_d(b.im, 0));
        if (mf.passes(d2f_scaled(f.x, bexp), d2f_scaled(f.y, bexp))) mf.take(f.x * s_inv, f.y * s_inv);
    }
    fold_max2(mb.best, mf.best, &ctl->c2, &ctl->fn);
    if (last_block(ctl) && threadIdx.x == 0) {
        volatile ExpmCtl *vc = ctl;
        double c2 = sqrt(__longlong_as_double((long long)vc->c2));
        double fn = sqrt(__longlong_as_double((long long)vc->fn));
        const double sc = pow2(bexp);
        c2 *= sc;
        fn *= sc;
        vc->terms = vc->terms + 1;
        if (vc->c1 + c2 <= tol * fn) vc->done = 1;
        else vc->c1 = c2;
        vc->c2 = 0ull;
        vc->fn = 0ull;
        __threadfence();
        vc->arrive = 0u;
    }
}

// A persistent grid, a slice per warp and turn.  Wider blocks keep more
// neighbouring slices on one SM at a time, whose L1 they share, but hand out
// the last slices more coarsely (16 against 8 warps: a term of 4.7 M rows 391 / 402
// us, 1.3 M 114 / 117, 361 k 46 / 44, 191 k 33 / 29).
struct SellGrid {
    int threads, blocks;
};
template <class K>
SellGrid sell_grid(K k, int64_t n, int (&resident)[2])
{
    const int wide = n >= (1 << 20), threads = wide ? 512 : 256, warps = threads / 32;
    return {threads, qs_persistent_grid(k, threads, ((n + 31) / 32 + warps - 1) / warps, resident[wide])};
}

template <class DV, bool XC>
int spmv_go(int64_t n, const int64_t *sptr, const int32_t *words, const void *data, const void *xs, void *y, cdbl a,
            int overwrite, const unsigned long long *xnorm, cudaStream_t st)
{
    static int resident[2] = {0, 0};
    auto k = sell_spmv_kernel<DV, XC>;
    const SellGrid g = sell_grid(k, n, resident);
    k<<<g.blocks, g.threads, 0, st>>>(n, sptr, words, data, xs, (double *)y, a, overwrite, xnorm);
    QS_CHECK(cudaGetLastError());
    return QS_OK;
}
template <class DV, bool XC>
int lz_go(const LzProduct &p, cudaStream_t st)
{
    static int resident[2] = {0, 0};
    auto k = sell_lz_kernel<DV, XC>;
    const SellGrid g = sell_grid(k, p.n, resident);
    k<<<g.blocks, g.threads, 0, st>>>(p, reinterpret_cast<const int64_t *>(p.indptr));
    QS_CHECK(cudaGetLastError());
    return QS_OK;
}
template <class DV>
int term_go(const LpTerm &a)
{
    static int resident[2] = {0, 0};
    auto k = taylor_sell_kernel<DV>;
    const SellGrid g = sell_grid(k, a.n, resident);
    k<<<g.blocks, g.threads, 0, a.st>>>(a.n, (const int64_t *)a.indptr, a.indices, a.data,
                                                    (const cpf *)a.Bin, (cpf *)a.Bout, a.F, a.mu0, a.coeff, a.j, a.tol,
                                                    (ExpmCtl *)a.ctl);
    QS_CHECK(cudaGetLastError());
    return QS_OK;
}

}  // namespace

int sell_spmv(int64_t n, const int64_t *sptr, const int32_t *words, const void *data, int dtype, const void *xs, int xc,
              void *y, cdbl a, int overwrite, const unsigned long long *xnorm, cudaStream_t st)
{
    if (dtype == QS_CPF8S) return xc ? spmv_go<cpf, true>(n, sptr, words, data, xs, y, a, overwrite, xnorm, st) : QS_ERR_ARG;
    return xc ? spmv_go<pf, true>(n, sptr, words, data, xs, y, a, overwrite, xnorm, st)
              : spmv_go<pf, false>(n, sptr, words, data, xs, y, a, overwrite, xnorm, st);
}

int sell_taylor_term(const LpTerm &a)
{
    if (a.nvec != 1 || a.btype != QS_CPF) return QS_ERR_ARG;
    return a.dtype == QS_CPF8S ? term_go<cpf>(a) : term_go<pf>(a);
}

int sell_lanczos(const LzProduct &p, int dtype, int cplx, cudaStream_t st)
{
    if (dtype == QS_CPF8S) return cplx ? lz_go<cpf, true>(p, st) : QS_ERR_ARG;
    return cplx ? lz_go<pf, true>(p, st) : lz_go<pf, false>(p, st);
}

// Groups of four slots per slice of 32 rows (int32 row pointers); most: the
// longest row (zeroed by the caller).
extern "C" int qs_sell_count(int64_t n, const int32_t *indptr, int64_t *groups, int *most, void *stream)
{
    if (n < 1 || !indptr || !groups || !most) return QS_ERR_ARG;
    sell_count_kernel<<<(unsigned)((n + 255) / 256), 256, 0, qs_stream(stream)>>>(n, indptr, groups, most);
    QS_CHECK(cudaGetLastError());
    return QS_OK;
}

// The sliced words of packed rows of at most 128 nonzeros.  sptr: groups before
// each slice, [slices + 1]; out: 128 words per group.
extern "C" int qs_sell_fill(int64_t n, const int32_t *indptr, const int32_t *words, const int64_t *sptr, int64_t groups,
                            int32_t *out, void *stream)
{
    if (n < 1 || groups < 0 || !indptr || !words || !sptr || !out) return QS_ERR_ARG;
    cudaStream_t st = qs_stream(stream);
    QS_CHECK(cudaMemsetAsync(out, 0xff, (size_t)groups * 512, st));
    const int64_t slices = (n + 31) / 32;
    sell_fill_kernel<<<(unsigned)((slices + 7) / 8), 256, 0, st>>>(n, indptr, words, sptr, (uint32_t *)out);
    QS_CHECK(cudaGetLastError());
    return QS_OK;
}
