// e^{aA} v of a small problem in one cooperative launch.
//
// The launch sequence of csrc/expm.cu runs one kernel per Taylor term: for a
// few thousand states a term is one or two microseconds of work in a launch of
// five to seven, and the launches left after a substep's stopping test fired
// still cost three each.  Here the whole evolution is one kernel: the grid
// (at most one block per SM) walks the terms itself, with one grid-wide barrier
// per term, and stops a substep where its test fires.  Same recurrence, shift,
// scaling and stopping test in the same arithmetic (float-pair products, F and
// the norms in IEEE double: csrc/expm_lp.cu).
//
// What bounds it is latency: a term is a chain of a column load, a gather, the
// row's sums, the block's norms and the barrier's round trip through L2, 5.1 us
// at 245 rows and 5.3 at 4752; past that the gathers add to it.  FP64
// instructions are kept off that chain where they can be: they cost an SM 16
// cycles each per warp and some 50 of latency.  A call with the stopping test
// before the last planned term, launch per term -> here, by events: XXZ L = 14
// (245 rows, 27 terms of 35) 274 -> 137 us; XXZ L = 20 (4752 rows, 54 of 80)
// 661 -> 285; Ising L = 18 (14541 rows, 274k nonzeros, 117 of 165) 1534 -> 908;
// Ising L = 20 (52377 rows, 1.1M nonzeros, 126 of 165) 2262 -> 1828.  Above
// 65535 rows, and 2.4 M entries, the launch shapes of csrc/expm_lp.cu are tuned or
// its resident warps hide the gathers better than one block per SM.  The rows on 128, 76 or
// 38 SMs instead of all 152: 294, 310, 385 us at 4752 rows, and more above.
//
// B changes hands between SMs inside the kernel: it is written through to L2
// and gathered past L1 (ld.cg); the matrix is read through L1, where each SM's
// rows stay from term to term.  The barrier counts arrivals upwards and gives
// up after a bounded number of polls; the launch is cooperative, so every block
// is resident and the wait ends.  Should it give up all the same, F is NaN, err
// is set in the control block and the input is kept for another way to evolve
// it (ExpmMultiplyParallel.settle).
#include "qs_common.cuh"
#include "expm_ctl.cuh"
#include "lp_lanes.cuh"

namespace {

constexpr int CT = 512;              // most threads per block
constexpr int CU = 4;                // gathers in flight per lane
constexpr int POLLS = 1 << 23;       // a few seconds: a poll is a trip to L2 and back

// Arrival count and the maxima of three reductions in turn; all zero between
// launches.  left: blocks that have finished; failed: whose wait gave up.
struct SmallSync {
    unsigned int arrive, left, failed, pad_;
    unsigned long long mb[3], mf[3];
};

struct SmallArgs {
    int n, lgG, s, m, polls;
    const int32_t *indptr, *indices;
    const void *data;
    cpf *B0, *B1;
    cdbl *F, *keep;            // keep: receives the input (nullable)
    const cdbl *coeff, *eta;
    cdbl mu;
    double tol;
    ExpmCtl *ctl;
    SmallSync *sync;
};

__device__ __forceinline__ cpf ld_shared_b(const cpf *p)
{
    const float4 v = __ldcg(reinterpret_cast<const float4 *>(p));
    return cpf{pf{v.x, v.y}, pf{v.z, v.w}};
}

// matrix values, kept in L1 from term to term
__device__ __forceinline__ pf ld_val(const pf *p) { return ModePF::ldS(p); }
__device__ __forceinline__ cpf ld_val(const cpf *p) { return ModePF::ldB(p); }

__device__ __forceinline__ unsigned long long max64(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

// Grid-wide maxima of two doubles >= 0 (as bits), reduction number e, which is
// also a barrier.  False when the wait gave up after `most` polls.  (Every block posting a word
// that all others poll, without atomics, measured twice as slow: 149 pollers on
// each of 149 lines.)
__device__ __forceinline__ bool grid_max2(SmallSync *sync, int most, unsigned &e, unsigned long long &a,
                                          unsigned long long &b)
{
    __shared__ unsigned long long sa[CT / 32], sb[CT / 32];
    __shared__ int ok;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int slot = e % 3, next = (e + 1) % 3;
    e++;
    for (int o = 16; o > 0; o >>= 1) {
        a = max64(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = max64(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    if (lane == 0) { sa[w] = a; sb[w] = b; }
    __syncthreads();                    // all of the block's stores are made, too
    if (threadIdx.x == 0) {
        for (int k = 1; k < nw; k++) { a = max64(a, sa[k]); b = max64(b, sb[k]); }
        if (a) atomicMax(&sync->mb[slot], a);
        if (b) atomicMax(&sync->mf[slot], b);
        // the next reduction's slot was read by every block before it arrived
        // at the barrier before this one
        if (blockIdx.x == 0) {
            sync->mb[next] = 0ull;
            sync->mf[next] = 0ull;
        }
        __threadfence();
        atomicAdd(&sync->arrive, 1u);
        const unsigned target = e * gridDim.x;
        int polls = 0;
        while ((int)(*((volatile unsigned int *)&sync->arrive) - target) < 0 && ++polls < most) {}
        __threadfence();
        ok = polls < most;
        sa[0] = __ldcg(&sync->mb[slot]);
        sb[0] = __ldcg(&sync->mf[slot]);
    }
    __syncthreads();
    a = sa[0];
    b = sb[0];
    const bool good = ok;
    __syncthreads();                    // before the next reduction's words
    return good;
}

// Whether c1 + c2 <= tol fn with c1, c2 and fn the roots of moduli squared
// (c1: of ca, or itself where first).  In FP32 unless the two sides are within
// a part in a hundred: both roots in FP64 take 0.5 us of latency, and every
// block waits for them on every term.
__device__ __forceinline__ bool stop_test(unsigned long long ca, bool first, unsigned long long mb,
                                          unsigned long long mf, double tol, int bexp)
{
    const double dc = __longlong_as_double((long long)ca), db = __longlong_as_double((long long)mb);
    const double df = __longlong_as_double((long long)mf);
    const float c1 = first ? d2f_scaled(dc, bexp) : sqrtf(d2f_scaled(dc, 0));
    const float lhs = c1 + sqrtf(d2f_scaled(db, 0)), rhs = d2f_scaled(tol, 0) * sqrtf(d2f_scaled(df, 0));
    if (lhs > 1.01f * rhs && lhs > 1e-18f) return false;
    const double sc = pow2(bexp);
    return (first ? dc : sqrt(dc) * sc) + sqrt(db) * sc <= tol * (sqrt(df) * sc);
}

template <class DV, int VM>
__global__ void __launch_bounds__(CT, 1) taylor_small_kernel(SmallArgs p)
{
    using M = ModePF;
    using S = pf;
    constexpr bool CODED = VM != 0;
    __shared__ DV s_tab[CODED ? QS_CODE_TABLE : 1];
    const DV *data = reinterpret_cast<const DV *>(p.data);
    const uint8_t *codes = nullptr;
    if constexpr (CODED) {
        for (int i = threadIdx.x; i < QS_CODE_TABLE; i += blockDim.x) s_tab[i] = ldv(data + i);
        codes = reinterpret_cast<const uint8_t *>(data + QS_CODE_TABLE);
        __syncthreads();
    }
    const int G = 1 << p.lgG, lane = threadIdx.x & (G - 1), comp = lane & 1;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    const int GPW = 32 >> p.lgG, gsub = (threadIdx.x & 31) >> p.lgG, warp = tid >> 5, nwarps = nthreads >> 5;
    const cdbl eta = *p.eta;
    const S mu_re = pair_rn_scaled(p.mu.x, 0), mu_im = pair_rn_scaled(p.mu.y, 0);
    unsigned e = 0;                     // reductions so far
    int nonconv = 0, bexp = 0;
    long long terms = 0;
    unsigned long long c1 = 0ull;       // bits of c1, or of its square after the first term
    bool ok = true;
    for (int step = 0; step <= p.s && ok; step++) {
        // F = eta F (not before the first substep), its norm, B0 = F 2^-bexp
        const bool scale = step > 0 && !(eta.x == 1.0 && eta.y == 0.0);
        unsigned long long mb = 0ull, mf = 0ull;
        for (int r = tid; r < p.n; r += nthreads) {
            const double2 v = __ldcg(reinterpret_cast<const double2 *>(p.F + r));
            double fx = v.x, fy = v.y;
            if (step == 0 && p.keep) __stcg(reinterpret_cast<double2 *>(p.keep + r), v);
            if (scale) {
                fx = eta.x * v.x - eta.y * v.y;
                fy = eta.x * v.y + eta.y * v.x;
                __stcg(reinterpret_cast<double2 *>(p.F + r), make_double2(fx, fy));
            }
            if (step < p.s) {
                // as fmax: a NaN counts as nothing
                const double h = hypot(fx, fy);
                if (h == h) mb = max64(mb, (unsigned long long)__double_as_longlong(h));
            }
        }
        if (step == p.s) break;
        ok = grid_max2(p.sync, p.polls, e, mb, mf);
        if (!ok) break;
        c1 = mb;
        bexp = scale_exp(__longlong_as_double((long long)c1));
        const double s_inv = pow2(-bexp);
        // this thread scaled these rows itself
        for (int r = tid; r < p.n; r += nthreads) {
            const double2 v = __ldcg(reinterpret_cast<const double2 *>(p.F + r));
            const pf re = pair_rn_scaled(v.x, bexp), im = pair_rn_scaled(v.y, bexp);
            __stcg(reinterpret_cast<float4 *>(p.B0 + r), make_float4(re.h, re.l, im.h, im.l));
        }
        mb = mf = 0ull;
        ok = grid_max2(p.sync, p.polls, e, mb, mf);
        bool done = false;
        for (int j = 0; j < p.m && ok && !done; j++) {
            const cpf *Bin = (j & 1) ? p.B1 : p.B0;
            cpf *Bout = (j & 1) ? p.B0 : p.B1;
            const cdbl cj = p.coeff[j];
            const S cf_re = pair_rn_scaled(cj.x, 0), cf_im = pair_rn_scaled(cj.y, 0);
            const S cm_re = M::sub(M::mul(cf_re, mu_re), M::mul(cf_im, mu_im));
            const S cm_im = M::add(M::mul(cf_re, mu_im), M::mul(cf_im, mu_re));
            const S cf_x = comp ? cf_im : M::neg(cf_im), cm_x = comp ? cm_im : M::neg(cm_im);
            mb = mf = 0ull;
            for (int rb = warp * GPW; rb < p.n; rb += nwarps * GPW) {
                const int r = rb + gsub;
                const bool valid = r < p.n, writer = valid && lane < 2;
                const int k0 = valid ? __ldg(p.indptr + r) : 0, k1 = valid ? __ldg(p.indptr + r + 1) : 0;
                cpf bo{M::zero(), M::zero()};
                double fv = 0.0;
                if (writer) {
                    bo = ld_shared_b(Bin + r);
                    fv = __ldcg(reinterpret_cast<const double *>(p.F + r) + comp);
                }
                S ar = M::zero(), ai = M::zero();
                for (int k = k0 + lane; k < k1; k += G * CU) {
                    int col[CU];
                    DV d[CU];
                    cpf b[CU];
#pragma unroll
                    for (int u = 0; u < CU; u++) {
                        const int kk = k + u * G;
                        const bool in = kk < k1;
                        col[u] = in ? __ldg(p.indices + kk) : 0;
                        if constexpr (CODED) d[u] = in ? s_tab[__ldg(codes + kk)] : vzero<DV>();
                        else d[u] = in ? ld_val(data + kk) : vzero<DV>();
                    }
#pragma unroll
                    for (int u = 0; u < CU; u++) b[u] = ld_shared_b(Bin + col[u]);
#pragma unroll
                    for (int u = 0; u < CU; u++)
                        if (k + u * G < k1) vmul_acc<M>(ar, ai, d[u], b[u]);
                }
                for (int o = G >> 1; o > 0; o >>= 1) {
                    ar = M::merge(ar, M::shfl_xor(ar, o));
                    ai = M::merge(ai, M::shfl_xor(ai, o));
                }
                // new term = cf (A B) - (cf mu) B, this lane's component
                const S acc_c = M::fin(comp ? ai : ar), acc_o = M::fin(comp ? ar : ai);
                const S bo_c = comp ? bo.im : bo.re, bo_o = comp ? bo.re : bo.im;
                const S mine = M::sub(M::add(M::mul(cf_re, acc_c), M::mul(cf_x, acc_o)),
                                      M::add(M::mul(cm_re, bo_c), M::mul(cm_x, bo_o)));
                double md = 0.0, fs = 0.0;
                if (writer) {
                    __stcg(reinterpret_cast<float2 *>(Bout + r) + comp, make_float2(mine.h, mine.l));
                    fv = M::add_to(fv, mine, bexp);
                    __stcg(reinterpret_cast<double *>(p.F + r) + comp, fv);
                    md = M::to_d(mine, 0);
                    fs = fv * s_inv;
                }
                double nb2 = __dmul_rn(md, md), f2 = __dmul_rn(fs, fs);
                nb2 = __dadd_rn(nb2, __shfl_xor_sync(0xffffffffu, nb2, 1));
                f2 = __dadd_rn(f2, __shfl_xor_sync(0xffffffffu, f2, 1));
                if (writer) {
                    if (nb2 == nb2) mb = max64(mb, (unsigned long long)__double_as_longlong(nb2));
                    if (f2 == f2) mf = max64(mf, (unsigned long long)__double_as_longlong(f2));
                }
            }
            ok = grid_max2(p.sync, p.polls, e, mb, mf);
            done = stop_test(c1, j == 0, mb, mf, p.tol, bexp);
            if (!done) c1 = mb;
            terms++;
        }
        if (p.m > 0 && !done) nonconv++;
    }
    // the last block to leave clears the words for the next launch; where a
    // barrier gave up it leaves no result rather than a wrong one
    __shared__ bool last, failed;
    __syncthreads();
    if (threadIdx.x == 0) {
        if (blockIdx.x == 0) {
            p.ctl->terms = terms;
            p.ctl->nonconv = nonconv;
        }
        if (!ok) atomicOr(&p.sync->failed, 1u);
        __threadfence();
        last = atomicAdd(&p.sync->left, 1u) + 1u == gridDim.x;
        __threadfence();
        failed = last && *((volatile unsigned int *)&p.sync->failed);
    }
    __syncthreads();
    if (!last) return;
    if (failed)
        for (int r = threadIdx.x; r < p.n; r += blockDim.x)
            p.F[r] = cdbl{__longlong_as_double(-1ll), __longlong_as_double(-1ll)};
    if (threadIdx.x == 0) {
        p.ctl->err = failed;
        for (int i = 0; i < 3; i++) p.sync->mb[i] = p.sync->mf[i] = 0ull;
        p.sync->arrive = p.sync->failed = 0u;
        __threadfence();
        p.sync->left = 0u;
    }
}

template <class DV, int VM>
int small_go(SmallArgs p, int64_t nnz, cudaStream_t st)
{
    // lanes per row until a row is one batch of gathers per lane, as the chip
    // holds; then the rows over all SMs (the epilogue's FP64 instructions cost
    // an SM the same for one active lane as for 32, so more lanes than that,
    // or fewer SMs, cost more than they save)
    int lg = 1;
    const int sms = qs_num_sms();
    while (lg < 4 && ((int64_t)p.n << lg) * CU < nnz && ((int64_t)p.n << (lg + 1)) <= (int64_t)sms * CT) lg++;
    p.lgG = lg;
    const int64_t lanes = (int64_t)p.n << lg;
    int64_t threads = ((lanes + sms - 1) / sms + 31) / 32 * 32;
    threads = threads < 64 ? 64 : (threads > CT ? CT : threads);
    const int64_t need = (lanes + threads - 1) / threads;
    const int blocks = (int)(need < sms ? need : sms);
    void *args[] = {&p};
    QS_CHECK(cudaLaunchCooperativeKernel((const void *)taylor_small_kernel<DV, VM>, dim3(blocks),
                                         dim3((unsigned)threads), args, 0, st));
    return QS_OK;
}

}  // namespace

extern "C" int qs_expm_small_sync_bytes() { return (int)sizeof(SmallSync); }

// qs_expm_multiply for one vector and float-pair storage (btype QS_CPF) of a
// small int32 matrix, as one cooperative launch: at most 2^17 rows and 2^30
// entries (an entry index and the lanes' stride fit an int); dtype
// QS_PF / QS_CPF or coded QS_PF8 / QS_CPF8.  sync: qs_expm_small_sync_bytes()
// of zeros before the first call, left zero; calls that share ctl, work or
// sync must not overlap.  The control block receives this call's terms and
// unconverged substeps (nothing is added up), and in its err word whether a
// grid barrier gave up after `polls` looks (a limit of the caller's for tests
// and watchdogs); F is NaN then, and keep (n elements, nullable) holds the input.
extern "C" int qs_expm_multiply_small_kept(int64_t n, int64_t nnz, const int32_t *indptr, const int32_t *indices,
                                           const void *data, int dtype, void *F, int s, int m_star, double tol,
                                           double mu_re, double mu_im, const void *coeff, const void *eta, void *work,
                                           void *ctl, void *sync, void *keep, int polls, void *stream)
{
    if (n < 1 || n > (1 << 17) || nnz < 0 || nnz > (1 << 30) || s < 1 || m_star < 0 || !indptr || !F || !coeff || !eta || !work || !ctl ||
        !sync || polls < 0 || polls > POLLS || (nnz > 0 && (!indices || !data)))
        return QS_ERR_ARG;
    SmallArgs p{(int)n, 1, s, m_star, polls, indptr, indices, data, (cpf *)work, (cpf *)work + n, (cdbl *)F,
                (cdbl *)keep, (const cdbl *)coeff, (const cdbl *)eta, cdbl{mu_re, mu_im}, tol, (ExpmCtl *)ctl, (SmallSync *)sync};
    switch (dtype) {
    case QS_PF: return small_go<pf, 0>(p, nnz, qs_stream(stream));
    case QS_CPF: return small_go<cpf, 0>(p, nnz, qs_stream(stream));
    case QS_PF8: return small_go<pf, 1>(p, nnz, qs_stream(stream));
    case QS_CPF8: return small_go<cpf, 1>(p, nnz, qs_stream(stream));
    default: return QS_ERR_ARG;
    }
}

extern "C" int qs_expm_small_polls() { return POLLS; }

// The same without a kept input, up to the largest number of polls.
extern "C" int qs_expm_multiply_small(int64_t n, int64_t nnz, const int32_t *indptr, const int32_t *indices,
                                      const void *data, int dtype, void *F, int s, int m_star, double tol,
                                      double mu_re, double mu_im, const void *coeff, const void *eta, void *work,
                                      void *ctl, void *sync, void *stream)
{
    return qs_expm_multiply_small_kept(n, nnz, indptr, indices, data, dtype, F, s, m_star, tol, mu_re, mu_im, coeff,
                                       eta, work, ctl, sync, nullptr, POLLS, stream);
}
