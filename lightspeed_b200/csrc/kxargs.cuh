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

// Work unit -> bra index and ket range. Units run chunk by chunk over all bras,
// the ket chunks with the largest bounds (the most quartets) first.
struct XUnit {
    int i, j0, j1;
};

__host__ __device__ __forceinline__ XUnit unit_of(const XGradArgs& A, unsigned unit)
{
    XUnit u;
    const unsigned nb = (unsigned) A.bn[0] + (unsigned) A.bn[1];
    const int c = (int) (unit / nb), bi = (int) (unit % nb);
    u.i = bi < A.bn[0] ? A.boff[0] + bi : A.boff[1] + (bi - A.bn[0]);
    const int nc0 = A.kn[0] ? (A.kn[0] - 1) / A.chunk + 1 : 0;
    const int s = c < nc0 ? 0 : 1, at = (c - (s ? nc0 : 0)) * A.chunk;
    const int left = A.kn[s] - at;
    u.j0 = A.koff[s] + at;
    u.j1 = u.j0 + (left < A.chunk ? left : A.chunk);
    return u;
}

// Kets per work unit and the number of units of nb bras and two ranges of kets: about
// `units` of them where there are that many pairs of pairs, a multiple of lo kets within
// [lo, hi], and more kets where the units would not fit the 32-bit queue (whose last draws
// go past the end, one per warp of the launch). Lists hold less than 2^31 - 32767 pairs (65535
// primitives), so whole ranges as chunks always fit.
struct XSplit {
    int chunk;
    unsigned nunit;
};
constexpr long kXMaxUnits = 0xffff0000L;

inline XSplit xgrad_split(long nb, long kn0, long kn1, long lo, long hi, long units)
{
    long chunk = nb * (kn0 + kn1) / units;
    chunk = (chunk + lo - 1) / lo * lo;
    chunk = chunk < lo ? lo : (chunk > hi ? hi : chunk);
    auto count = [&] { return nb * ((kn0 + chunk - 1) / chunk + (kn1 + chunk - 1) / chunk); };
    while (count() > kXMaxUnits) chunk *= 2;
    const long whole = kn0 > kn1 ? kn0 : kn1;
    if (chunk > whole && chunk > hi) chunk = whole;
    return XSplit{(int) chunk, (unsigned) count()};
}

template <int L1, int L2>
void launch_xgrad_12(Context* ctx, const XGradArgs& A, int L3, int L4);

} // namespace lsjk
