// Arguments of the K gradient over unique quartets (kxgrad.cu) and the
// declaration of its per-class launchers.
#pragma once
#include "kargs.cuh"

namespace lsjk {

// One (bra class | ket class). The pairs of the pair list stand in its order
// (class, bound descending) with the shell of larger angular momentum first;
// a class (L1 >= L2) is up to two ranges of them, the list's (L1, L2) and
// (L2, L1).
struct XGradArgs {
    // per pair (a b): exponent sum q, h K_ab / q with h = 1/2 if a = b, centre P, A - B,
    // r = (exponent of b) / q (so P - A = -r (A - B)), Cartesian offsets and primitives
    // of a and b, the larger primitive index, and the Schwarz bound
    const double *q, *kab, *P[3], *CD[3], *r;
    const int *cc, *cd, *pa, *pb, *pm;
    const float* bound;
    int boff[2], bn[2];       // bra ranges
    int koff[2], kn[2];       // ket ranges
    BasisView b;
    const double* D;          // symmetric density (Cartesian, ld)
    int ld;
    const double* dblk;       // max|D block| per primitive pair (nprim x nprim)
    double* G;                // ncopy copies of the gradient, ng numbers each
    int ncopy, ng;
    const KScalars* sc;       // max|D| and the K-invert bound threshold
    float thr;                // thresp
    int chunk;                // kets per work unit
    unsigned nunit;           // work units: bras x ket chunks
    unsigned* queue;
    int* status;
    const double* rys;        // FP64 Rys table block of the rule one quantum up
    const double *asym_t, *asym_w;
    int nbin;
    double tmax;
    int nterm;
    double alpha[4], omega[4];
};

template <int L1, int L2>
void launch_xgrad_12(Context* ctx, const XGradArgs& A, int L3, int L4);

} // namespace lsjk
