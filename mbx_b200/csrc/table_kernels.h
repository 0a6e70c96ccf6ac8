// What the host code hands to the table-driven kernels (table_kernels.cu).
#pragma once
#include <cuda_runtime.h>

// The term table of a polynomial in the w variables (term_table.cuh), its
// coefficients c = F a, and the rows of W (w = W x - w0) and of its transpose:
// entry +-(column + 1).
struct PolyTable {
    const int4* terms;
    const double* tcoef;
    long nterms;
    int pairs;
    const double* coef;
    const int *wrow, *w, *wtrow, *wt;
    const double* w0;
};

// A polynomial over caller-supplied variables.
int mbx_launch_poly_table(long nd, int nvars, const double* x, double* g, double* e, const PolyTable& P, int sms,
                          cudaStream_t s);

struct AdjointTable {
    const int4* terms;
    const double* tcoef;
    int nterms, nhalf, nvars, ncoef, ncw;
    const int2* half;
    const unsigned* pair;     // half-monomials of the terms, in the order of the first one
    const int* term;          // the terms in that order
    const int *first, *ftrow, *ftk;   // first term of every coefficient; rows of F transposed
    const double* ftf;
};

// Coefficient adjoint over n-mers whose w variables are in wv; work:
// (mbx_coef_adjoint_blocks + 1) * nterms + ncw doubles.
int mbx_coef_adjoint_blocks(const AdjointTable& P, int sms);
int mbx_launch_coef_adjoint(const double* wv, int count, const AdjointTable& P, double* work, double* out, int sms,
                            cudaStream_t s);

// Polynomials of at most this many terms have their adjoint in one kernel
// (holder_dcoef_small_kernel).
#define MBX_SMALL_TERMS 32
