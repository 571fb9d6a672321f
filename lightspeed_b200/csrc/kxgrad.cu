// K gradient of the fully symmetric call (IntBox::exchangeGrad with D13symm,
// D24symm and Dsame: one symmetric density D, the RHF gradient; reference
// src/cpp/intbox/cpu/exchange_grad.cpp:17-470) over unique quartets.
//
//   G = sum over ordered quartets (1,2,3,4) of D13 d(12|34)/dR D24
//
// The eight orders of a quartet share their integral derivatives, and their
// density products are only two, so with (a b| and |c d) running over the
// unique pairs of the pair list
//   G = sum over bra and ket pairs  4 h_ab h_cd (D_ac D_bd + D_bc D_ad)
//                                   (d/dA + d/dB) (ab|cd),   h = 1/2 if a = b.
// Both orders of the two pairs occur as (bra, ket), so each quartet needs the
// derivatives at its bra's centres alone: nothing is scattered to the ket's
// atoms, and the six sums of a bra stay in registers while its kets pass by.
// Against a quartet per ordered (1,2,3,4) with derivatives at three centres
// (kgrad.cu, kept for densities that differ or lack the symmetry) this is a
// quarter of the quartets, each evaluated twice with fewer derivatives.
//
// The reference screens a quartet by its representative's density block,
//   bound_ab bound_cd max|D(max(a, b), max(c, d))| >= thresp,
// which leaves a few per cent of the pairs of pairs of a large molecule. A
// warp owns a bra; its lanes test 32 kets at a time (bound order, so a chunk
// ends early) and queue the passing ones in shared memory, and a full queue
// of 32 runs as one batch, a quartet per lane, whatever the pass rate was.
//
// Bound by the FP64 pipe and its latency at 8 warps per multiprocessor (the
// straight-line quartets use 128-255 registers). Measured, the K gradient alone
// through the host API, against the general routine on the same density (one
// quartet per ordered (1,2,3,4) and warp): C10H22/cc-pVDZ with a density of
// converged extent 20.1 against 371 ms, (H2O)2/cc-pVTZ 2.5 against 40.2 ms.
#include <algorithm>
#include <atomic>
#include "engine.cuh"
#include "kxargs.cuh"
#include "lsjk_device.cuh"
#include "hermite.cuh"   // cart_lx/ly/lz

#include LSJK_XG_HEADER   // the straight-line quartets of this bra class

namespace lsjk {

namespace {

constexpr int kXThreads = 128, kXWarps = kXThreads / 32;
constexpr double kTwoPi52X = 34.986836655249725693;   // 2 pi^(5/2)

__device__ __forceinline__ double xwarp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The bra of a work unit, the same on every lane.
struct XBra {
    double a2, b2;             // 2 alpha, 2 beta
    double p, ip, kab;
    double P[3], PA[3], AB[3];
    int ca, cb;                // Cartesian offsets of a and b
    int atomA, atomB, rmax;    // atoms; the larger primitive index
    float bound;
};

__device__ __forceinline__ XBra load_bra(const XGradArgs& A, int i)
{
    XBra b;
    const int pa = A.pa[i], pb = A.pb[i];
    const double alpha = A.b.e[pa], beta = A.b.e[pb];
    b.a2 = 2.0 * alpha;
    b.b2 = 2.0 * beta;
    b.p = A.q[i];
    b.ip = 1.0 / b.p;
    b.kab = A.kab[i];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        b.P[d] = A.P[d][i];
        b.AB[d] = A.CD[d][i];
        b.PA[d] = -A.r[i] * b.AB[d];
    }
    b.ca = A.cc[i];
    b.cb = A.cd[i];
    b.atomA = A.b.atom[pa];
    b.atomB = A.b.atom[pb];
    b.rmax = max(pa, pb);
    b.bound = A.bound[i];
    return b;
}

// Adds the bra's sums to this CTA's copy of G.
__device__ __forceinline__ void add_bra(const XGradArgs& A, const XBra& b, int lane, const double gA[3],
                                        const double gB[3])
{
    double* G = A.G + (long) (blockIdx.x % A.ncopy) * A.ng;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double sa = xwarp_sum(gA[d]), sb = xwarp_sum(gB[d]);
        if (lane == 0) {
            if (sa != 0.0) atomicAdd(&G[3 * b.atomA + d], sa);
            if (sb != 0.0) atomicAdd(&G[3 * b.atomB + d], sb);
        }
    }
}

// A quartet per lane.
template <int L1, int L2, int L3, int L4>
__global__ void __launch_bounds__(kXThreads) k_xgrad(const __grid_constant__ XGradArgs A)
{
    constexpr int NR = (L1 + L2 + L3 + L4 + 1) / 2 + 1;
    constexpr int N1 = ncart_of(L1), N2 = ncart_of(L2), N3 = ncart_of(L3), N4 = ncart_of(L4);
    extern __shared__ __align__(128) unsigned char xg_smem[];
    double* tab = reinterpret_cast<double*>(xg_smem);
    __shared__ __align__(8) uint64_t mbar;
    __shared__ int queue_all[kXWarps][64];
    if (!stage_bulk(tab, A.rys, (unsigned) (rys_block<double>(NR, A.nbin) * sizeof(double)), &mbar, A.status)) return;
    const int lane = threadIdx.x & 31;
    int* pend = queue_all[threadIdx.x >> 5];
    const float thre = A.sc->thre12;
    const double dmax = __longlong_as_double((long long) A.sc->dmax_bits);
    const double thr = (double) A.thr, bscale = A.nbin / A.tmax;
    for (;;) {
        unsigned unit = 0;
        if (lane == 0) unit = atomicAdd(A.queue, 1u);
        unit = __shfl_sync(0xffffffffu, unit, 0);
        if (unit >= A.nunit) break;
        const XUnit U = unit_of(A, unit);
        const float bi = A.bound[U.i];
        if (bi < thre || (double) (bi * A.bound[U.j0]) * dmax < thr) continue;   // bound order: nothing passes
        const XBra B = load_bra(A, U.i);
        const double* drow = A.dblk + (long) B.rmax * A.b.nprim;
        double gA[3] = {0, 0, 0}, gB[3] = {0, 0, 0};
        int npend = 0;

        auto quartet = [&](int j) {
            const double q = A.q[j], iq = 1.0 / q, rr = A.r[j];
            double CD[3], QC[3], PQ[3], RR = 0.0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                CD[d] = A.CD[d][j];
                QC[d] = -rr * CD[d];
                PQ[d] = B.P[d] - A.P[d][j];
                RR = fma(PQ[d], PQ[d], RR);
            }
            const int cc = A.cc[j], cd = A.cd[j];
            double Dac[N1 * N3], Dbd[N2 * N4], Dbc[N2 * N3], Dad[N1 * N4];
#pragma unroll
            for (int x = 0; x < N1; ++x) {
                const double* row = A.D + (long) (B.ca + x) * A.ld;
#pragma unroll
                for (int y = 0; y < N3; ++y) Dac[x * N3 + y] = row[cc + y];
#pragma unroll
                for (int y = 0; y < N4; ++y) Dad[x * N4 + y] = row[cd + y];
            }
#pragma unroll
            for (int x = 0; x < N2; ++x) {
                const double* row = A.D + (long) (B.cb + x) * A.ld;
#pragma unroll
                for (int y = 0; y < N3; ++y) Dbc[x * N3 + y] = row[cc + y];
#pragma unroll
                for (int y = 0; y < N4; ++y) Dbd[x * N4 + y] = row[cd + y];
            }
            const double p = B.p;
            const double rs = rsqrt(p + q);
            const double ipq = rs * rs;
            const double rho = p * q * ipq;
            const double pref = 4.0 * kTwoPi52X * (B.kab * A.kab[j]) * rs;   // (kab fields: h K_ab / p)
#pragma unroll 1
            for (int tm = 0; tm < A.nterm; ++tm) {
                double d2 = 1.0, f = A.alpha[tm] * pref;
                if (A.omega[tm] != -1.0) {
                    const double w2 = A.omega[tm] * A.omega[tm];
                    d2 = w2 / (rho + w2);
                    f *= sqrt(d2);
                }
                double t2[NR], w[NR];
                rys_eval<NR, double>(rho * d2 * RR, tab, A.nbin, A.tmax, bscale, A.asym_t, A.asym_w, t2, w);
                // one root after another: slot 0 is the root in use and the rest shift down,
                // so the arrays keep static indices and the code one copy of the root
#pragma unroll 1
                for (int r = 0; r < NR; ++r) {
                    const double u = t2[0] * d2 * ipq, qu = q * u, pu = p * u;
                    XG<L1, L2, L3, L4>::template run<double>(
                        B.PA[0] - qu * PQ[0], B.PA[1] - qu * PQ[1], B.PA[2] - qu * PQ[2], QC[0] + pu * PQ[0],
                        QC[1] + pu * PQ[1], QC[2] + pu * PQ[2], 0.5 * u, 0.5 * B.ip * (1.0 - qu),
                        0.5 * iq * (1.0 - pu), B.AB[0], B.AB[1], B.AB[2], CD[0], CD[1], CD[2], f * w[0], B.a2, B.b2,
                        Dac, Dbd, Dbc, Dad, gA, gB);
#pragma unroll
                    for (int k = 0; k + 1 < NR; ++k) {
                        t2[k] = t2[k + 1];
                        w[k] = w[k + 1];
                    }
                }
            }
        };

        for (int js = U.j0;; js += 32) {
            const bool more = js < U.j1 && (double) (bi * A.bound[js]) * dmax >= thr;
            if (more) {
                const int j = js + lane;
                bool pass = false;
                if (j < U.j1) {
                    const float bj = A.bound[j];
                    pass = bj >= thre && (double) (bi * bj) * drow[A.pm[j]] >= thr;
                }
                const unsigned m = __ballot_sync(0xffffffffu, pass);
                if (pass) pend[npend + __popc(m & ((1u << lane) - 1u))] = j;
                npend += __popc(m);
            }
            if (more && npend < 32) continue;
            // a full batch, or the rest of the chunk
            __syncwarp();
            const int nrun = min(npend, 32);
            const int jq = lane < nrun ? pend[lane] : -1;
            const int jr = lane + 32 < npend ? pend[lane + 32] : 0;
            __syncwarp();
            if (lane + 32 < npend) pend[lane] = jr;
            npend -= nrun;
            if (jq >= 0) quartet(jq);
            __syncwarp();
            if (!more && npend == 0) break;
        }
        add_bra(A, B, lane, gA, gB);
    }
}

// Per-warp shared tables of a quartet of the heavy classes.
template <int L1, int L2, int L3, int L4>
struct XWarpTab {
    static constexpr int NR = (L1 + L2 + L3 + L4 + 1) / 2 + 1;
    static constexpr int MA = L1 + L2 + 1, MC = L3 + L4, S2 = L2 + 1, S3 = L3 + 1, S4 = L4 + 1;
    static constexpr int SG = (L1 + 1) * S2 * S3 * S4;
    double H[NR][3][L2 + 2][MA + 1][MC + 1];   // every root's integrals after the transfer to centre 2
    double T[3][SG][4];                        // one root's integrals and their derivatives at a and b
    double Dac[ncart_of(L1) * ncart_of(L3)], Dbd[ncart_of(L2) * ncart_of(L4)];
    double Dbc[ncart_of(L2) * ncart_of(L3)], Dad[ncart_of(L1) * ncart_of(L4)];
};

// Warps per CTA of the quartet-per-warp kernel: four while their tables leave room for two
// CTAs per multiprocessor, else two ((ff|ff): 75 KB per warp).
template <int L1, int L2, int L3, int L4>
constexpr int xwarp_warps()
{
    return 4 * sizeof(XWarpTab<L1, L2, L3, L4>) <= 110 * 1024 ? 4 : 2;
}

// A quartet per warp, for the classes whose straight-line quartet would not fit registers:
//   * one (root, direction) per lane runs the vertical recursion and the transfer to centre 2;
//   * per root, one (direction, a, b, {value, d/dA, d/dB}) row per lane: the derivative is
//     formed first (2 alpha H(a+1) - a H(a-1), likewise in b), then the row goes to centre 4;
//   * the contraction as jobs (i1, i3, a range of i2) over the lanes, i4 innermost.
// Screens and work units are those of k_xgrad.
template <int L1, int L2, int L3, int L4>
__global__ void __launch_bounds__(kXThreads) k_xgrad_warp(const __grid_constant__ XGradArgs A)
{
    using Tab = XWarpTab<L1, L2, L3, L4>;
    constexpr int NR = Tab::NR, MA = Tab::MA, MC = Tab::MC, S2 = Tab::S2, S3 = Tab::S3, S4 = Tab::S4;
    constexpr int N1 = ncart_of(L1), N2 = ncart_of(L2), N3 = ncart_of(L3), N4 = ncart_of(L4);
    constexpr int NO = N1 * N3, NPART = NO >= 32 ? 1 : (N2 < 32 / NO ? N2 : 32 / NO);
    constexpr int NJOB = NO * NPART;
    extern __shared__ __align__(128) unsigned char xg_smem[];
    Tab& S = reinterpret_cast<Tab*>(xg_smem)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const float thre = A.sc->thre12;
    const double dmax = __longlong_as_double((long long) A.sc->dmax_bits);
    const double thr = (double) A.thr, bscale = A.nbin / A.tmax;
    const int rl = lane < 3 * NR ? lane / 3 : 0, dl = lane % 3;   // this lane's root and direction
    for (;;) {
        unsigned unit = 0;
        if (lane == 0) unit = atomicAdd(A.queue, 1u);
        unit = __shfl_sync(0xffffffffu, unit, 0);
        if (unit >= A.nunit) break;
        const XUnit U = unit_of(A, unit);
        const float bi = A.bound[U.i];
        if (bi < thre || (double) (bi * A.bound[U.j0]) * dmax < thr) continue;
        const XBra B = load_bra(A, U.i);
        const double* drow = A.dblk + (long) B.rmax * A.b.nprim;
        double gA[3] = {0, 0, 0}, gB[3] = {0, 0, 0};
        const double PAd = dl == 0 ? B.PA[0] : (dl == 1 ? B.PA[1] : B.PA[2]);
        const double ABd = dl == 0 ? B.AB[0] : (dl == 1 ? B.AB[1] : B.AB[2]);
        for (int js = U.j0; js < U.j1; js += 32) {
            if ((double) (bi * A.bound[js]) * dmax < thr) break;
            bool pass = false;
            if (js + lane < U.j1) {
                const float bj = A.bound[js + lane];
                pass = bj >= thre && (double) (bi * bj) * drow[A.pm[js + lane]] >= thr;
            }
            unsigned m = __ballot_sync(0xffffffffu, pass);
            while (m) {
                const int j = js + __ffs(m) - 1;
                m &= m - 1;
                const double q = A.q[j], iq = 1.0 / q, rr = A.r[j];
                double CD[3], PQ[3], RR = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    CD[d] = A.CD[d][j];
                    PQ[d] = B.P[d] - A.P[d][j];
                    RR = fma(PQ[d], PQ[d], RR);
                }
                const int cc = A.cc[j], cd = A.cd[j];
                __syncwarp();   // the previous quartet's tables have been read
                for (int k = lane; k < N1 * N3; k += 32) S.Dac[k] = A.D[(long) (B.ca + k / N3) * A.ld + cc + k % N3];
                for (int k = lane; k < N2 * N4; k += 32) S.Dbd[k] = A.D[(long) (B.cb + k / N4) * A.ld + cd + k % N4];
                for (int k = lane; k < N2 * N3; k += 32) S.Dbc[k] = A.D[(long) (B.cb + k / N3) * A.ld + cc + k % N3];
                for (int k = lane; k < N1 * N4; k += 32) S.Dad[k] = A.D[(long) (B.ca + k / N4) * A.ld + cd + k % N4];
                const double p = B.p;
                const double rs = rsqrt(p + q);
                const double ipq = rs * rs;
                const double rho = p * q * ipq;
                const double pref = 4.0 * kTwoPi52X * (B.kab * A.kab[j]) * rs;
                const double PQd = dl == 0 ? PQ[0] : (dl == 1 ? PQ[1] : PQ[2]);
                const double QCd = -rr * (dl == 0 ? CD[0] : (dl == 1 ? CD[1] : CD[2]));
#pragma unroll 1
                for (int tm = 0; tm < A.nterm; ++tm) {
                    double d2 = 1.0, f = A.alpha[tm] * pref;
                    if (A.omega[tm] != -1.0) {
                        const double w2 = A.omega[tm] * A.omega[tm];
                        d2 = w2 / (rho + w2);
                        f *= sqrt(d2);
                    }
                    __syncwarp();
                    if (lane < 3 * NR) {
                        double t2, w;
                        rys_root(rho * d2 * RR, A.rys, NR, rl, A.nbin, A.tmax, bscale, A.asym_t, A.asym_w, t2, w);
                        const double u = t2 * d2 * ipq, qu = q * u, pu = p * u;
                        const double b00 = 0.5 * u, b10 = 0.5 * B.ip * (1.0 - qu), b01 = 0.5 * iq * (1.0 - pu);
                        const double c00 = PAd - qu * PQd, d00 = QCd + pu * PQd;
                        double I[MA + 1][MC + 1];
                        I[0][0] = dl == 2 ? f * w : 1.0;
#pragma unroll
                        for (int a = 0; a < MA; ++a) I[a + 1][0] = c00 * I[a][0] + (a ? a * b10 * I[a - 1][0] : 0.0);
#pragma unroll
                        for (int c = 0; c < MC; ++c)
#pragma unroll
                            for (int a = 0; a <= MA; ++a) {
                                double v = d00 * I[a][c];
                                if (c) v += c * b01 * I[a][c - 1];
                                if (a) v += a * b00 * I[a - 1][c];
                                I[a][c + 1] = v;
                            }
                        // transfer to centre 2 in place: H(a, b+1) = H(a+1, b) + (A - B) H(a, b)
#pragma unroll
                        for (int b = 0; b <= L2 + 1; ++b) {
#pragma unroll
                            for (int a = 0; a <= MA - b; ++a)
#pragma unroll
                                for (int c = 0; c <= MC; ++c) S.H[rl][dl][b][a][c] = I[a][c];
#pragma unroll
                            for (int a = 0; a + 1 <= MA - b; ++a)
#pragma unroll
                                for (int c = 0; c <= MC; ++c) I[a][c] = fma(ABd, I[a][c], I[a + 1][c]);
                        }
                    }
                    __syncwarp();
#pragma unroll 1
                    for (int r = 0; r < NR; ++r) {
                        for (int row = lane; row < 9 * (L1 + 1) * S2; row += 32) {
                            const int kind = row % 3, d = (row / 3) % 3, ab = row / 9, a = ab / S2, b = ab % S2;
                            const double CDd = d == 0 ? CD[0] : (d == 1 ? CD[1] : CD[2]);
                            auto& H = S.H[r][d];
                            double V[MC + 1];
                            if (kind == 0) {
#pragma unroll
                                for (int c = 0; c <= MC; ++c) V[c] = H[b][a][c];
                            } else if (kind == 1) {
#pragma unroll
                                for (int c = 0; c <= MC; ++c)
                                    V[c] = B.a2 * H[b][a + 1][c] - (a ? a * H[b][a - 1][c] : 0.0);
                            } else {
#pragma unroll
                                for (int c = 0; c <= MC; ++c)
                                    V[c] = B.b2 * H[b + 1][a][c] - (b ? b * H[b - 1][a][c] : 0.0);
                            }
                            double* o = &S.T[d][ab * S3 * S4][kind];
#pragma unroll
                            for (int e = 0; e <= L4; ++e) {
#pragma unroll
                                for (int c = 0; c <= L3; ++c) o[(c * S4 + e) * 4] = V[c];
#pragma unroll
                                for (int c = 0; c + 1 <= MC - e; ++c) V[c] = fma(CDd, V[c], V[c + 1]);
                            }
                        }
                        __syncwarp();
#pragma unroll 1
                        for (int job = lane; job < NJOB; job += 32) {
                            const int o13 = job / NPART, part = job % NPART;
                            const int i1 = o13 / N3, i3 = o13 % N3;
                            const double dac = S.Dac[o13];
                            const int x1 = cart_lx(L1, i1), y1 = cart_ly(L1, i1), z1 = cart_lz(L1, i1);
                            const int x3 = cart_lx(L3, i3), y3 = cart_ly(L3, i3), z3 = cart_lz(L3, i3);
#pragma unroll 1
                            for (int i2 = part * N2 / NPART; i2 < (part + 1) * N2 / NPART; ++i2) {
                                const double dbc = S.Dbc[i2 * N3 + i3];
                                const int x2 = cart_lx(L2, i2), y2 = cart_ly(L2, i2), z2 = cart_lz(L2, i2);
                                const double(*tx)[4] = &S.T[0][((x1 * S2 + x2) * S3 + x3) * S4];
                                const double(*ty)[4] = &S.T[1][((y1 * S2 + y2) * S3 + y3) * S4];
                                const double(*tz)[4] = &S.T[2][((z1 * S2 + z2) * S3 + z3) * S4];
                                int i4 = 0;
#pragma unroll
                                for (int j4 = 0; j4 <= L4; ++j4)
#pragma unroll
                                    for (int z4 = 0; z4 <= j4; ++z4, ++i4) {
                                        const double W = fma(dac, S.Dbd[i2 * N4 + i4], dbc * S.Dad[i1 * N4 + i4]);
                                        const double* X = tx[L4 - j4];
                                        const double* Y = ty[j4 - z4];
                                        const double* Z = tz[z4];
                                        const double wx = W * X[0], wz = W * Z[0];
                                        const double yz = wz * Y[0], xz = wx * Z[0], xy = wx * Y[0];
                                        gA[0] = fma(X[1], yz, gA[0]);
                                        gA[1] = fma(Y[1], xz, gA[1]);
                                        gA[2] = fma(Z[1], xy, gA[2]);
                                        gB[0] = fma(X[2], yz, gB[0]);
                                        gB[1] = fma(Y[2], xz, gB[1]);
                                        gB[2] = fma(Z[2], xy, gB[2]);
                                    }
                            }
                        }
                        __syncwarp();   // the table is rewritten by the next root
                    }
                }
            }
        }
        add_bra(A, B, lane, gA, gB);
    }
}

template <int L1, int L2, int L3, int L4>
void launch_one(Context* ctx, const XGradArgs& A0)
{
    XGradArgs A = A0;
    constexpr bool lane = XG<L1, L2, L3, L4>::lane;
    const long nb = (long) A.bn[0] + A.bn[1], nk = (long) A.kn[0] + A.kn[1];
    if (nb == 0 || nk == 0) return;
    // a few units per warp of the GPU, [32, 2048] kets each (a partial last batch of a unit
    // wastes lanes) for a quartet per lane and [4, 256] for a quartet per warp
    const XSplit split =
        xgrad_split(nb, A.kn[0], A.kn[1], lane ? 32 : 4, lane ? 2048 : 256, 16L * ctx->nsm * kXWarps);
    A.chunk = split.chunk;
    A.nunit = split.nunit;
    size_t smem;
    if constexpr (lane)
        smem = (size_t) rys_block<double>((L1 + L2 + L3 + L4 + 1) / 2 + 1, A.nbin) * sizeof(double);
    else
        smem = xwarp_warps<L1, L2, L3, L4>() * sizeof(XWarpTab<L1, L2, L3, L4>);
    constexpr int warps = lane ? kXWarps : xwarp_warps<L1, L2, L3, L4>();
    const unsigned grid = (unsigned) std::min<long>(((long) A.nunit + warps - 1) / warps, 8L * ctx->nsm);
    auto run = [&](auto kern) {
        // the shared-memory opt-in is a per-device function attribute: set it once per device
        static std::atomic<unsigned long long> devices{0};
        const unsigned long long bit = 1ull << (ctx->device & 63);
        if (smem > 32 * 1024 && !(devices.load(std::memory_order_acquire) & bit)) {
            LSJK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
            devices.fetch_or(bit, std::memory_order_acq_rel);
        }
        kern<<<grid, 32 * warps, smem, ctx->stream>>>(A);
        LSJK_CUDA(cudaGetLastError());
        ctx->stats.kernel_launches++;
    };
    if constexpr (lane)
        run(k_xgrad<L1, L2, L3, L4>);
    else
        run(k_xgrad_warp<L1, L2, L3, L4>);
}

} // namespace

// The ket classes of bra class (L1, L2); this unit holds one bra class.
template <int L1, int L2>
void launch_xgrad_12(Context* ctx, const XGradArgs& A, int L3, int L4)
{
    switch (10 * L3 + L4) {
    case 0: launch_one<L1, L2, 0, 0>(ctx, A); break;
    case 10: launch_one<L1, L2, 1, 0>(ctx, A); break;
    case 11: launch_one<L1, L2, 1, 1>(ctx, A); break;
    case 20: launch_one<L1, L2, 2, 0>(ctx, A); break;
    case 21: launch_one<L1, L2, 2, 1>(ctx, A); break;
    case 22: launch_one<L1, L2, 2, 2>(ctx, A); break;
    case 30: launch_one<L1, L2, 3, 0>(ctx, A); break;
    case 31: launch_one<L1, L2, 3, 1>(ctx, A); break;
    case 32: launch_one<L1, L2, 3, 2>(ctx, A); break;
    case 33: launch_one<L1, L2, 3, 3>(ctx, A); break;
    default: throw Error(LSJK_ENOTSUPP, "K gradient: shell above f");
    }
}
template void launch_xgrad_12<LSJK_L1, LSJK_L2>(Context*, const XGradArgs&, int, int);

} // namespace lsjk
