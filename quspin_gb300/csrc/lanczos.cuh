// Shared by the Lanczos kernels (csrc/lanczos.cu) and their fused product
// (csrc/spmv_lp.cu): the run's control words and the block reductions.
#pragma once
#include "qs_common.cuh"

struct LzCtl {
    int done;      // b[i] < eps was seen
    int m_eff;     // number of valid Lanczos vectors
};

// Control words of a whole run on the device: LzCtl, then the arrival counter
// of the reductions that finish in their own launch.
struct LzRunCtl {
    int done, m_eff;
    unsigned int arrive;
    int pad_;
};

// One product r = A q - b v with the dot product <q, r>.
struct LzProduct {
    int64_t n;
    const int32_t *indptr, *indices;
    const void *data;          // float-pair values or the code table
    const void *xs;            // q 2^xexp as float pairs
    int xexp;
    const double *q, *v, *b;   // v null in the first step
    double *r, *partial, *alpha;
    LzRunCtl *ctl;
};

int spmv_lanczos(const LzProduct &p, int pdtype, int cplx, int group, cudaStream_t st);

namespace {

__device__ __forceinline__ double wsum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double block_sum(double v)
{
    __shared__ double sh[32];
    v = wsum(v);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
    if (w == 0) {
        t = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
        t = wsum(t);
    }
    return t;   // valid in thread 0
}

enum LzFinish {
    LZ_SUM,       // out = sum
    LZ_BETA,      // out = sqrt(sum); below eps: done, m_eff = i
    LZ_BEFORE,    // state = {sum, 0}: the squared norm before a Gram-Schmidt pass
    LZ_PASS       // the pass's verdict in state (see lz_verdict), then as LZ_BETA
};

// Pass control of the adaptive reorthogonalisation.  state[0]: squared norm
// of r before the last pass; state[1]: 1 once a pass kept at least 1/sqrt(2)
// of the norm (then r is orthogonal to the rows to working precision and
// the remaining passes return at once).
__device__ __forceinline__ void lz_verdict(double s, double *state)
{
    if (s >= 0.5 * state[0]) state[1] = 1.0;
    else state[0] = s;
}

// Sum over the grid of one value per thread, finished by the last block to
// arrive: the block partials in a fixed order, so the result does not depend
// on timing.  Saves the launch (about 3 us) of a finishing kernel.
__device__ __forceinline__ void lz_block_finish(double v, double *partial, double *out, int what, double eps, int i,
                                                double *state, LzRunCtl *ctl)
{
    __shared__ bool last;
    const double s = block_sum(v);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(&ctl->arrive, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;
    const volatile double *vp = partial;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) t += vp[k];
    t = block_sum(t);
    if (threadIdx.x == 0) {
        if (what == LZ_SUM) *out = t;
        if (what == LZ_BEFORE) {
            state[0] = t;
            state[1] = 0.0;
        }
        if (what == LZ_PASS) lz_verdict(t, state);
        if (what == LZ_BETA || what == LZ_PASS) {
            const double b = sqrt(t);
            *out = b;
            if (b < eps) {
                ctl->done = 1;
                ctl->m_eff = i;
            }
        }
        ctl->arrive = 0u;
    }
}

}  // namespace
