// Symmetry maps and orbit walks of the basis kernels (csrc/basis.cu).
//
// A map permutes the sites of a state (and may invert them).  Where the
// permutation moves its bits by at most four different distances -- chain and
// lattice translations by two, a chain reflection by one after a bit reversal,
// an inversion by none -- it is applied in registers as masked shifts;
// otherwise from byte-indexed tables in shared memory.  The masked form is two
// or three integer instructions per distance; a table costs a scattered
// shared-memory load per byte (about 3.5 bank conflicts each).
//
// The group's elements are visited in odometer order (the last map runs
// fastest).  The walk keeps only the state in registers and the element's
// digits as packed bytes: the phase and the fermion sign are formed afterwards
// for the one element that matters, not along the way.  Up to four maps of at
// most 256 powers take this form (nested loops, unrolled by template); more
// maps or longer periods take the odometer with its position in local memory.
#pragma once
#include "qs_common.cuh"

#define QS_MAXMAPS 32
#define QS_MAXGRP 4       // masked shifts per map
#define QS_MAXPAIR 16     // factors of a map's fermion sign

// The maps, in the kernel's parameters (constant memory).
template <typename S>
struct SymParams {
    int N, nmaps, fermion, L, nbytes;
    int fast;                        // maps walked by the nested loops (0: the odometer)
    int pers[QS_MAXMAPS];
    int step[QS_MAXMAPS];
    int qcap[QS_MAXMAPS];            // digits covered by the quick representative test
    S flip[QS_MAXMAPS];
    S gmask[QS_MAXMAPS][QS_MAXGRP];  // masked shifts, left by gshift (right where negative)
    int8_t gshift[QS_MAXMAPS][QS_MAXGRP];
    int8_t ngrp[QS_MAXMAPS];         // number of masked shifts (0: the byte tables)
    int8_t rev[QS_MAXMAPS];          // reverse the N bits first
    int8_t npair[QS_MAXMAPS];        // sign factors (-1: the later-and-lower masks)
    const S *tab;                    // masks | sign factors | byte tables
    unsigned pair_off, lut_off;
    const double *ph_re, *ph_im, *cost;
};

// The maps and their tables, staged in shared memory.
template <typename S>
struct SymView {
    const SymParams<S> &P;
    const S *ll;     // nmaps * N (fermion)
    const S *pair;   // nmaps * QS_MAXPAIR * 2 (fermion)
    const S *lut;    // nmaps * nbytes * 256
};

// Copies the first nelem elements of the map tables into shared memory (the
// byte tables come last and are left out of nelem when no map reads them).
template <typename S>
__device__ __forceinline__ SymView<S> stage_tables(const SymParams<S> &P, S *smem, size_t nelem)
{
    for (size_t i = threadIdx.x; i < nelem; i += blockDim.x) smem[i] = P.tab[i];
    __syncthreads();
    return SymView<S>{P, smem, smem + P.pair_off, smem + P.lut_off};
}

__device__ __forceinline__ uint32_t rev_bits(uint32_t s, int N) { return __brev(s) >> (32 - N); }
__device__ __forceinline__ uint64_t rev_bits(uint64_t s, int N)
{
    return (uint64_t)__brevll((unsigned long long)s) >> (64 - N);
}
__device__ __forceinline__ int pop_bits(uint32_t s) { return __popc(s); }
__device__ __forceinline__ int pop_bits(uint64_t s) { return __popcll((unsigned long long)s); }
// a shift whose bits never leave the word, as a rotation
__device__ __forceinline__ uint32_t move_bits(uint32_t x, int sh) { return __funnelshift_l(x, x, sh); }
__device__ __forceinline__ uint64_t move_bits(uint64_t x, int sh) { return sh >= 0 ? x << sh : x >> -sh; }

// image of s under map k
template <typename S>
__device__ __forceinline__ S map_bits(const SymView<S> &V, int k, S s)
{
    S out;
    const int ng = V.P.ngrp[k];
    if (ng) {
        const S t = V.P.rev[k] ? rev_bits(s, V.P.N) : s;
        out = move_bits((S)(t & V.P.gmask[k][0]), V.P.gshift[k][0]);
        if (ng > 1) out |= move_bits((S)(t & V.P.gmask[k][1]), V.P.gshift[k][1]);
        if (ng > 2) {
            out |= move_bits((S)(t & V.P.gmask[k][2]), V.P.gshift[k][2]);
            out |= move_bits((S)(t & V.P.gmask[k][3]), V.P.gshift[k][3]);
        }
    } else {
        const S *lk = V.lut + (size_t)k * V.P.nbytes * 256;
        out = 0;
        for (int b = 0; b < V.P.nbytes; b++) out |= lk[b * 256 + (int)((s >> (8 * b)) & 0xff)];
    }
    return out ^ V.P.flip[k];
}

// parity of the fermion reordering of map k on s: the number of pairs of
// occupied sites whose order it reverses
template <typename S>
__device__ __forceinline__ int map_parity(const SymView<S> &V, int k, S s)
{
    int inv = 0;
    const int np = V.P.npair[k];
    if (np >= 0) {
        const S *p = V.pair + (size_t)k * QS_MAXPAIR * 2;
        for (int i = 0; i < np; i++) inv ^= pop_bits((S)(s & p[2 * i])) & pop_bits((S)(s & p[2 * i + 1]));
    } else {
        const S *ll = V.ll + (size_t)k * V.P.N;
        S m = s;
        while (m) {
            int pos;
            if (sizeof(S) == 8) pos = 63 - __clzll((long long)m);
            else pos = 31 - __clz((int)m);
            m &= ~((S)1 << pos);
            inv += pop_bits((S)(s & ll[V.P.N - 1 - pos]));
        }
    }
    return inv & 1;
}

template <typename S>
__device__ __forceinline__ S map_state(const SymView<S> &V, int k, S s, int &sign)
{
    if (V.P.fermion && map_parity(V, k, s)) sign = -sign;
    return map_bits(V, k, s);
}

// Visits the images of s, digits d of map D running over lim[D] values (the
// last map fastest), as f(image, packed digits); stops when f returns false.
template <int K, int D, typename S, class F>
__device__ __forceinline__ bool orbit_walk(const SymView<S> &V, const int *lim, S s, uint32_t digits, F &f)
{
    if constexpr (D == K) {
        return f(s, digits);
    } else {
        const int per = lim[D];
        if (D == K - 1 && V.P.ngrp[D] == 2 && !V.P.rev[D]) {
            // the fastest map of most groups, a translation: its two masked
            // shifts stay in registers and the loop is straight code
            const S m0 = V.P.gmask[D][0], m1 = V.P.gmask[D][1], fl = V.P.flip[D];
            const int s0 = V.P.gshift[D][0], s1 = V.P.gshift[D][1];
#pragma unroll 4
            for (int i = 0; i < per; i++) {
                if (!f(s, digits | ((uint32_t)i << (8 * D)))) return false;
                s = (move_bits((S)(s & m0), s0) | move_bits((S)(s & m1), s1)) ^ fl;
            }
            return true;
        }
        for (int i = 0;;) {
            if (!orbit_walk<K, D + 1>(V, lim, s, digits | ((uint32_t)i << (8 * D)), f)) return false;
            if (++i >= per) return true;
            s = map_bits(V, D, s);
        }
    }
}

template <typename S, class F>
__device__ __forceinline__ bool orbit_visit(const SymView<S> &V, const int *lim, S s, F &f)
{
    switch (V.P.fast) {
    case 1: return orbit_walk<1, 0>(V, lim, s, 0u, f);
    case 2: return orbit_walk<2, 0>(V, lim, s, 0u, f);
    case 3: return orbit_walk<3, 0>(V, lim, s, 0u, f);
    default: return orbit_walk<4, 0>(V, lim, s, 0u, f);
    }
}

// phase index and sign of the element with the given digits on s
template <typename S>
__device__ __forceinline__ void element_phase(const SymView<S> &V, S s, uint32_t digits, int &sign, int &phase)
{
    sign = 1;
    phase = 0;
    if (!digits) return;
    for (int d = 0; d < V.P.fast; d++) {
        const int n = (digits >> (8 * d)) & 0xff;
        phase = (phase + n * V.P.step[d]) % V.P.L;
        if (V.P.fermion)
            for (int i = 0; i < n; i++) s = map_state(V, d, s, sign);
    }
}

// state of the odometer over the group (any number of maps and powers)
template <typename S>
struct Odometer {
    S cur[QS_MAXMAPS + 1];
    int sg[QS_MAXMAPS + 1], ph[QS_MAXMAPS + 1], idx[QS_MAXMAPS];
    __device__ void start(const SymView<S> &V, S s)
    {
        for (int d = 0; d <= V.P.nmaps; d++) { cur[d] = s; sg[d] = 1; ph[d] = 0; }
        for (int d = 0; d < V.P.nmaps; d++) idx[d] = 0;
    }
    // advances to the next element; false after the last
    __device__ bool next(const SymView<S> &V)
    {
        const int K = V.P.nmaps;
        for (int d = K - 1; d >= 0; d--) {
            if (++idx[d] < V.P.pers[d]) {
                cur[d + 1] = map_state(V, d, cur[d + 1], sg[d + 1]);
                const int p = ph[d + 1] + V.P.step[d];
                ph[d + 1] = p >= V.P.L ? p - V.P.L : p;
                for (int e = d + 1; e < K; e++) { cur[e + 1] = cur[d + 1]; sg[e + 1] = sg[d + 1]; ph[e + 1] = ph[d + 1]; }
                return true;
            }
            idx[d] = 0;
        }
        return false;
    }
};

// norm of s as a representative (0 if not a representative)
template <typename S>
__device__ __forceinline__ double check_state(const SymView<S> &V, S s)
{
    if (V.P.nmaps == 0) return 1.0;
    double norm = 0.0;
    if (V.P.fast) {
        auto f = [&](S t, uint32_t digits) {
            if (t > s) return false;
            if (t == s) {
                int sg, ph;
                element_phase(V, s, digits, sg, ph);
                norm += sg * V.P.cost[ph];
            }
            return true;
        };
        if (!orbit_visit(V, V.P.pers, s, f)) return 0.0;
    } else {
        Odometer<S> o;
        o.start(V, s);
        do {
            const S t = o.cur[V.P.nmaps];
            if (t > s) return 0.0;
            if (t == s) norm += o.sg[V.P.nmaps] * V.P.cost[o.ph[V.P.nmaps]];
        } while (o.next(V));
    }
    const double r = floor(norm + 0.5);
    return r < 0.5 ? 0.0 : r;
}

// false when one of the first few elements (qcap digits of each map) already
// takes s to a larger state; the rest pass on to check_state
template <typename S>
__device__ __forceinline__ bool may_represent(const SymView<S> &V, S s)
{
    if (!V.P.fast) return true;
    bool ok = true;
    auto f = [&](S t, uint32_t) {
        ok = ok && t <= s;
        return true;
    };
    orbit_visit(V, V.P.qcap, s, f);
    return ok;
}

// largest orbit element, with the digits (g, nullable), sign and phase index
// of the first element in odometer order that reaches it
template <typename S>
__device__ __forceinline__ S ref_state(const SymView<S> &V, S s, int *g, int &sign_out, int &phase_out)
{
    const int K = V.P.nmaps;
    sign_out = 1;
    phase_out = 0;
    if (g) for (int d = 0; d < K; d++) g[d] = 0;
    if (K == 0) return s;
    S best = s;
    if (V.P.fast) {
        uint32_t at = 0;
        auto f = [&](S t, uint32_t digits) {
            if (t > best) { best = t; at = digits; }
            return true;
        };
        orbit_visit(V, V.P.pers, s, f);
        element_phase(V, s, at, sign_out, phase_out);
        if (g) for (int d = 0; d < K; d++) g[d] = (at >> (8 * d)) & 0xff;
    } else {
        Odometer<S> o;
        o.start(V, s);
        do {
            const S t = o.cur[K];
            if (t > best) {
                best = t;
                sign_out = o.sg[K];
                phase_out = o.ph[K];
                if (g) for (int d = 0; d < K; d++) g[d] = o.idx[d];
            }
        } while (o.next(V));
    }
    return best;
}
