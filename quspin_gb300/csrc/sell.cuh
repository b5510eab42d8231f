// The sliced form of a packed operand and its single-vector kernels
// (csrc/sell.cu), called from the product, the Taylor term and the Lanczos run.
#pragma once
#include "expm_ctl.cuh"
#include "lanczos.cuh"

#define QS_PF8S 10     // QS_PF8P in slices of 32 rows (see csrc/sell.cu)
#define QS_CPF8S 11    // the same for QS_CPF8P

static inline bool sell_type(int dtype) { return dtype == QS_PF8S || dtype == QS_CPF8S; }

int sell_spmv(int64_t n, const int64_t *sptr, const int32_t *words, const void *data, int dtype, const void *xs, int xc,
              void *y, cdbl a, int overwrite, const unsigned long long *xnorm, cudaStream_t st);
int sell_taylor_term(const LpTerm &a);
int sell_lanczos(const LzProduct &p, int dtype, int cplx, cudaStream_t st);
