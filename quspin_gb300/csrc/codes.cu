// Value codes: an array with at most 256 distinct doubles (or complex doubles)
// as a sorted table and one byte per value.
//
// Two streaming passes and no sort.  The first collects the distinct values in
// a hash table, each block in shared memory before it adds its own to the one
// in global memory; one block then sorts the few that there are; the second
// pass looks every value up.  A complex value is coded by the codes of its two
// parts; the pairs that occur are marked in a bitmap between the passes.
// Bound by the reading of the values (twice, complex three times) where they
// exceed L2.  Measured, sorting -> here, the read of the count included: 159 M real
// values 40.2 -> 1.54 ms, 52 k 0.41 -> 0.11 ms; a process's first call, which
// loaded the sort's kernels, 2.96 s -> 3 ms.
#include "qs_common.cuh"

namespace {

constexpr int SLOTS = 1024, MOST = 256;

struct CodeState {
    int over;                              // more than 256 distinct values, or a NaN
    int distinct;
    int count[2];                          // distinct real and imaginary parts
    unsigned long long key[2][SLOTS];      // hash tables of ordered keys, 0 for none
    unsigned char code[2][SLOTS];          // rank of the slot's key
    unsigned int pairs[65536 / 32];        // pairs of codes that occur
    unsigned char pair_code[65536];
};

// Keys in the order of the doubles (both zeros the same), never 0 for a number
__device__ __forceinline__ unsigned long long ordered(double x)
{
    unsigned long long u = (unsigned long long)__double_as_longlong(x);
    if ((u << 1) == 0ull) u = 0ull;
    return u ^ ((unsigned long long)((long long)u >> 63) | 0x8000000000000000ull);
}
__device__ __forceinline__ double unordered(unsigned long long k)
{
    return __longlong_as_double((long long)(k >> 63 ? k ^ 0x8000000000000000ull : ~k));
}
__device__ __forceinline__ bool is_nan(double x)
{
    return ((unsigned long long)__double_as_longlong(x) << 1) > 0xffe0000000000000ull;
}
__device__ __forceinline__ int home(unsigned long long k) { return (int)((k * 0x9e3779b97f4a7c15ull) >> 54); }

// Adds a key to a table; returns whether it is new.  *full is set when the
// table has no place for it.
__device__ __forceinline__ bool insert(unsigned long long *table, unsigned long long k, bool *full)
{
    int s = home(k);
    for (int i = 0; i < SLOTS; i++, s = (s + 1) & (SLOTS - 1)) {
        unsigned long long cur = *((volatile unsigned long long *)(table + s));
        if (cur == k) return false;
        if (cur == 0ull) {
            cur = atomicCAS(table + s, 0ull, k);
            if (cur == 0ull) return true;
            if (cur == k) return false;
        }
    }
    *full = true;
    return false;
}

// NC: parts per value
template <int NC>
__global__ void __launch_bounds__(256) codes_collect_kernel(int64_t count, const double *__restrict__ src, CodeState *st)
{
    __shared__ unsigned long long table[NC][SLOTS];
    __shared__ int n[NC], over;
    for (int i = threadIdx.x; i < NC * SLOTS; i += blockDim.x) table[0][i] = 0ull;
    if (threadIdx.x < NC) n[threadIdx.x] = 0;
    if (threadIdx.x == 0) over = *((volatile int *)&st->over);
    __syncthreads();
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    bool full = false;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += 4 * step) {
        double x[4][NC];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int64_t at = i + u * step < count ? i + u * step : i;
            if constexpr (NC == 2) {
                const double2 v = __ldcs(reinterpret_cast<const double2 *>(src) + at);
                x[u][0] = v.x;
                x[u][1] = v.y;
            } else {
                x[u][0] = __ldcs(src + at);
            }
        }
        if (*((volatile int *)&over)) break;
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int c = 0; c < NC; c++) {
                if (is_nan(x[u][c])) full = true;
                else if (insert(table[c], ordered(x[u][c]), &full) && atomicAdd(&n[c], 1) >= MOST) full = true;
                if (full) over = 1;
            }
    }
    __syncthreads();
    if (over) {
        if (threadIdx.x == 0) st->over = 1;
        return;
    }
    for (int i = threadIdx.x; i < NC * SLOTS; i += blockDim.x) {
        const unsigned long long k = table[0][i];
        if (!k || *((volatile int *)&st->over)) continue;
        const int c = i / SLOTS;
        if (insert(st->key[c], k, &full) && atomicAdd(&st->count[c], 1) >= MOST) full = true;
        if (full) st->over = 1;
    }
}

// One block: ranks of the keys; for real values the table itself
__global__ void __launch_bounds__(SLOTS) codes_rank_kernel(int nc, CodeState *st, double *__restrict__ vals)
{
    __shared__ unsigned long long list[MOST];
    __shared__ int n;
    if (st->over) return;
    for (int c = 0; c < nc; c++) {
        if (threadIdx.x == 0) n = 0;
        __syncthreads();
        const unsigned long long k = st->key[c][threadIdx.x];
        if (k) list[atomicAdd(&n, 1)] = k;
        __syncthreads();
        if (k) {
            int rank = 0;
            for (int i = 0; i < n; i++) rank += list[i] < k;
            st->code[c][threadIdx.x] = (unsigned char)rank;
            if (nc == 1) vals[rank] = unordered(k);
        }
        if (threadIdx.x == 0 && nc == 1) st->distinct = n;
        __syncthreads();
    }
}

__device__ __forceinline__ unsigned lookup(const unsigned long long *table, const unsigned char *code, double x)
{
    const unsigned long long k = ordered(x);
    int s = home(k);
    while (table[s] != k && table[s] != 0ull) s = (s + 1) & (SLOTS - 1);      // at most 256 of the slots are taken
    return code[s];
}

// What the second pass does with a value's code(s)
enum CodePass { CODES_REAL, CODES_MARK, CODES_PAIR };

template <int PASS>
__global__ void __launch_bounds__(256) codes_encode_kernel(int64_t count, const double *__restrict__ src, CodeState *st,
                                                           unsigned char *__restrict__ out)
{
    constexpr int NC = PASS == CODES_REAL ? 1 : 2;
    __shared__ unsigned long long table[NC][SLOTS];
    __shared__ unsigned char code[NC][SLOTS];
    __shared__ unsigned int seen[PASS == CODES_MARK ? 65536 / 32 : 1];
    if (st->over) return;
    for (int i = threadIdx.x; i < NC * SLOTS; i += blockDim.x) {
        table[0][i] = st->key[0][i];
        code[0][i] = st->code[0][i];
    }
    if constexpr (PASS == CODES_MARK)
        for (int i = threadIdx.x; i < 65536 / 32; i += blockDim.x) seen[i] = 0u;
    __syncthreads();
    // four values in a row per thread: one store of their bytes
    for (int64_t i = 4 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x); i < count; i += 4 * (int64_t)gridDim.x * blockDim.x) {
        const int m = count - i < 4 ? (int)(count - i) : 4;
        unsigned word = 0u;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (u >= m) break;
            unsigned e;
            if constexpr (NC == 1) {
                e = lookup(table[0], code[0], __ldcs(src + i + u));
            } else {
                const double2 v = __ldcs(reinterpret_cast<const double2 *>(src) + i + u);
                e = lookup(table[0], code[0], v.x) << 8 | lookup(table[1], code[1], v.y);
                if constexpr (PASS == CODES_MARK) {
                    const unsigned bit = 1u << (e & 31u);
                    if (!(*((volatile unsigned int *)&seen[e >> 5]) & bit)) atomicOr(&seen[e >> 5], bit);
                } else {
                    e = st->pair_code[e];
                }
            }
            word |= e << 8 * u;
        }
        if constexpr (PASS != CODES_MARK) {
            if (m == 4) *reinterpret_cast<unsigned *>(out + i) = word;
            else
                for (int u = 0; u < m; u++) out[i + u] = (unsigned char)(word >> 8 * u);
        }
    }
    if constexpr (PASS == CODES_MARK) {
        __syncthreads();
        for (int i = threadIdx.x; i < 65536 / 32; i += blockDim.x)
            if (seen[i]) atomicOr(&st->pairs[i], seen[i]);
    }
}

// One block: the pairs in order of their codes, the order of (real, imaginary)
__global__ void __launch_bounds__(1024) codes_pairs_kernel(CodeState *st, double *__restrict__ vals)
{
    __shared__ int before[1024];
    __shared__ double part[2][MOST];
    if (st->over) return;
    for (int i = threadIdx.x; i < 2 * SLOTS; i += 1024) {
        const unsigned long long k = st->key[0][i];
        if (k) part[i / SLOTS][st->code[0][i]] = unordered(k);
    }
    unsigned int w[2] = {st->pairs[2 * threadIdx.x], st->pairs[2 * threadIdx.x + 1]};
    const int mine = __popc(w[0]) + __popc(w[1]);
    before[threadIdx.x] = mine;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int add = threadIdx.x >= o ? before[threadIdx.x - o] : 0;
        __syncthreads();
        before[threadIdx.x] += add;
        __syncthreads();
    }
    const int total = before[1023];
    if (total > MOST) {
        if (threadIdx.x == 0) st->over = 1;
        return;
    }
    int at = before[threadIdx.x] - mine;
    for (int h = 0; h < 2; h++)
        for (; w[h]; w[h] &= w[h] - 1, at++) {
            const int e = 64 * threadIdx.x + 32 * h + __ffs(w[h]) - 1;
            st->pair_code[e] = (unsigned char)at;
            vals[2 * at] = part[0][e >> 8];
            vals[2 * at + 1] = part[1][e & 255];
        }
    if (threadIdx.x == 0) st->distinct = total;
}

}  // namespace

extern "C" int qs_value_codes_state_bytes() { return (int)sizeof(CodeState); }

// The table (256 doubles, or real and imaginary parts in turn for cplx, zeros
// past the last) and the code bytes of count values.  state:
// qs_value_codes_state_bytes() of device memory, whose first two words receive
// whether the values cannot be coded (more than 256 distinct ones, or a NaN) and
// the number of distinct values.
extern "C" int qs_value_codes(int64_t count, const double *src, int cplx, double *vals, unsigned char *codes, void *state,
                              void *stream)
{
    if (count < 1 || !src || !vals || !codes || !state || ((uintptr_t)codes & 3u)) return QS_ERR_ARG;
    cudaStream_t cs = qs_stream(stream);
    CodeState *st = (CodeState *)state;
    QS_CHECK(cudaMemsetAsync(st, 0, sizeof(CodeState), cs));
    QS_CHECK(cudaMemsetAsync(vals, 0, sizeof(double) * MOST * (cplx ? 2 : 1), cs));
    // a block's table costs as much as some thousand values
    const int64_t b = (count + 4095) / 4096, cap = (int64_t)qs_num_sms() * 8;
    const int blocks = (int)(b > cap ? cap : b);
    if (cplx) codes_collect_kernel<2><<<blocks, 256, 0, cs>>>(count, src, st);
    else codes_collect_kernel<1><<<blocks, 256, 0, cs>>>(count, src, st);
    codes_rank_kernel<<<1, SLOTS, 0, cs>>>(cplx ? 2 : 1, st, vals);
    if (cplx) {
        codes_encode_kernel<CODES_MARK><<<blocks, 256, 0, cs>>>(count, src, st, codes);
        codes_pairs_kernel<<<1, 1024, 0, cs>>>(st, vals);
        codes_encode_kernel<CODES_PAIR><<<blocks, 256, 0, cs>>>(count, src, st, codes);
    } else {
        codes_encode_kernel<CODES_REAL><<<blocks, 256, 0, cs>>>(count, src, st, codes);
    }
    QS_CHECK(cudaGetLastError());
    return QS_OK;
}
