// The J kernel: one template per Hermite class pair (LB|LK), instantiated in
// jinst.cu (compiled once per LB) so the classes build in parallel.
#pragma once
#include "engine.cuh"
#include "lsjk_device.cuh"
#include "generated/jquartets.cuh"
#include "jargs.cuh"
#include <atomic>

namespace lsjk {




// One J quartet (bra pair in registers, ket record r whose header q, Q the
// caller has already loaded) accumulated into jp, for the NG densities of the
// record (the Hermite integrals R_tuv are shared).
template <int LB, int LK, int NG>
__device__ __forceinline__ void j_quartet64(const JArgs& A, int g0, const double* tab, double p, double Px, double Py,
                                            double Pz, double q, double Qx, double Qy, double Qz,
                                            const double* __restrict__ r, double (*jp)[nherm_of(LB)])
{
    constexpr int L = LB + LK, HK = nherm_of(LK);
    const double X = Px - Qx, Y = Py - Qy, Z = Pz - Qz;
    const double R2 = X * X + Y * Y + Z * Z;
    const double rs = rsqrt(p + q);
    const double rho = p * q * (rs * rs);
    for (int tm = 0; tm < A.nterm; ++tm) {
        double d2 = 1.0, f = A.alpha[tm] * rs;
        if (!(A.bare >> tm & 1)) {
            const double om = A.omega[tm], w2 = om * om;
            d2 = w2 / (rho + w2);
            f *= sqrt(d2);
        }
        const double rhoe = rho * d2;
        double F[L + 1];
        boys_eval<L, double>(rhoe * R2, tab, F);
        double a[L + 1];
        const double m2r = -2.0 * rhoe;
        double pw = f;
#pragma unroll
        for (int n = 0; n <= L; ++n) {
            a[n] = pw * F[n];
            pw *= m2r;
        }
#pragma unroll
        for (int g = 0; g < NG; ++g)
            if (g0 + g < A.ng) jq_dispatch<LB, LK>(a, X, Y, Z, r + 4 + (g0 + g) * HK, jp[g]);
    }
}

// Densities per CTA for a bra class: the batched kernel keeps NG x HB FP64
// accumulators per thread (and as many FP32 ones), so the heavy bra classes
// take fewer densities per CTA (more CTA z-slices over the same ket records)
// instead of spilling.
template <int LB>
__host__ __device__ constexpr int j_batch() { return nherm_of(LB) <= 4 ? kJBatch : (nherm_of(LB) <= 10 ? 2 : 1); }

// Start of the last bin of the Boys table: from here on (the bin next to the
// switch to the asymptotic form, and the asymptotic region itself) the FP32
// path evaluates the Boys function in FP64 by its asymptotic form.
constexpr float kBoysSwitch32 = (float) (LSJK_BOYS_TMAX - LSJK_BOYS_TMAX / LSJK_BOYS_NBIN);

// The same quartet in FP32 (geometry differences formed in FP64, everything
// else in FP32 except the Boys function at T >= kBoysSwitch32, which is
// evaluated in FP64 by its asymptotic form), added to the FP64 accumulators.
template <int LB, int LK, int NG>
__device__ __forceinline__ void j_quartet32(const JArgs& A, int g0, const float* tab, float p,
                                            double Px, double Py, double Pz, double Qx, double Qy, double Qz,
                                            const float* __restrict__ r32, double (*jp)[nherm_of(LB)])
{
    constexpr int L = LB + LK, HB = nherm_of(LB), HK = nherm_of(LK);
    const float q = r32[0];
    const double Xd = Px - Qx, Yd = Py - Qy, Zd = Pz - Qz;
    const float X = (float) Xd, Y = (float) Yd, Z = (float) Zd;
    const float R2 = X * X + Y * Y + Z * Z;
    const float rs = rsqrtf(p + q);
    const float rho = p * q * (rs * rs);
    float jq[NG][HB];
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int t = 0; t < HB; ++t) jq[g][t] = 0.0f;
    for (int tm = 0; tm < A.nterm; ++tm) {
        float d2 = 1.0f, f = A.alphaf[tm] * rs;
        if (!(A.bare >> tm & 1)) {
            const float w2 = A.omegaf[tm] * A.omegaf[tm];
            d2 = w2 / (rho + w2);
            f *= sqrtf(d2);
        }
        const float rhoe = rho * d2;
        float F[L + 1];
        const float T = rhoe * R2;
        if (T < kBoysSwitch32) {
            boys_eval<L, float>(T, tab, F);
        } else {
            boys_asym_f64_to_f32<L>((double) rhoe * (Xd * Xd + Yd * Yd + Zd * Zd), F);
        }
        float a[L + 1];
        const float m2r = -2.0f * rhoe;
        float pw = f;
#pragma unroll
        for (int n = 0; n <= L; ++n) {
            a[n] = pw * F[n];
            pw *= m2r;
        }
#pragma unroll
        for (int g = 0; g < NG; ++g)
            if (g0 + g < A.ng) jq_dispatch<LB, LK>(a, X, Y, Z, r32 + 4 + (g0 + g) * HK, jq[g]);
    }
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int t = 0; t < HB; ++t) jp[g][t] += (double) jq[g][t];
}

template <int LB, int LK, int NG>
__global__ void __launch_bounds__(kJThreads) k_coulomb(JArgs A)
{
    constexpr int HB = nherm_of(LB), HK = nherm_of(LK);
    const int S = 4 + A.slots * HK;              // doubles (floats) per ket record
    __shared__ __align__(128) double tab[LSJK_BOYS_NBIN * 8];
    __shared__ __align__(128) float tab32[LSJK_BOYS_NBIN * 8];
    __shared__ __align__(8) uint64_t mbar[2];
    const int nb = *A.nbra, nk = *A.nket;
    const int g0 = blockIdx.z * NG;   // the densities g0 .. g0 + NG - 1 of the build
    const int i0 = blockIdx.x * kJThreads;
    const int j0 = blockIdx.y * A.chunk;
    if (i0 >= nb || j0 >= nk) return;
    const float B0 = A.bbound[i0];
    if (B0 * A.kbound[j0] < A.thresp) return;
    if (!stage_bulk(tab, A.boys, sizeof(tab), &mbar[0], A.status)) return;
    if (A.mixed && !stage_bulk(tab32, A.boys32, sizeof(tab32), &mbar[1], A.status)) return;

    const int i = i0 + threadIdx.x;
    const bool act = i < nb;
    double p = 1.0, Px = 0.0, Py = 0.0, Pz = 0.0;
    float Bi = 0.0f;
    if (act) {
        p = A.bgeom[4L * i];
        Px = A.bgeom[4L * i + 1];
        Py = A.bgeom[4L * i + 2];
        Pz = A.bgeom[4L * i + 3];
        Bi = A.bbound[i];
    }
    const float p32 = (float) p;
    const float thr_dp = A.mixed ? A.thredp : 0.0f;
    double jp[NG][HB];
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int t = 0; t < HB; ++t) jp[g][t] = 0.0;
    long nq = 0, nq32 = 0;
    const int nd = min(NG, A.ng - g0);   // statistics count density-quartets
    const int j1 = min(j0 + A.chunk, nk);
    // the next ket's bound and record header are loaded one iteration ahead, so
    // their latency overlaps the current quartet (all lanes read the same ket)
    float Bn = A.kbound[j0];
    double qn, Qxn, Qyn, Qzn;
    {
        const double* r = A.krec + (long) j0 * S;
        qn = r[0];
        Qxn = r[1];
        Qyn = r[2];
        Qzn = r[3];
    }
    for (int j = j0; j < j1; ++j) {
        const float Bj = Bn;
        const double qk = qn, Qx = Qxn, Qy = Qyn, Qz = Qzn;
        if (B0 * Bj < A.thresp) break;
        if (j + 1 < j1) {
            const double* rn = A.krec + (long) (j + 1) * S;
            Bn = A.kbound[j + 1];
            qn = rn[0];
            Qxn = rn[1];
            Qyn = rn[2];
            Qzn = rn[3];
        }
        const float est = Bi * Bj;
        const bool pass = act && est >= A.thresp;
        // one precision per warp and ket: FP64 while any lane's estimate reaches thredp
        // (those lanes need it; the others get FP64 too rather than a second, FP32
        // pass of the warp over the same ket), FP32 after. The kets are in bound
        // order, so the warp switches once.
        const bool dp = __any_sync(0xffffffffu, pass && est >= thr_dp);
        const double* r = A.krec + (long) j * S;
        if (dp) {
            if (pass) {
                nq += nd;
                j_quartet64<LB, LK, NG>(A, g0, tab, p, Px, Py, Pz, qk, Qx, Qy, Qz, r, jp);
            }
        } else if (__any_sync(0xffffffffu, pass)) {
            if (pass) {
                nq32 += nd;
                j_quartet32<LB, LK, NG>(A, g0, tab32, p32, Px, Py, Pz, Qx, Qy, Qz, A.krec32 + (long) j * S, jp);
            }
        }
    }
    if (act) {
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int t = 0; t < HB; ++t) {
                const double v = jp[g][t];
                if (v != 0.0 && g0 + g < A.ng) atomicAdd(&A.jbra[(g0 + g) * A.jbra_stride + (long) i * HB + t], v);
            }
    }
    // quartet counts for the statistics
    for (int o = 16; o > 0; o >>= 1) {
        nq += __shfl_xor_sync(0xffffffffu, nq, o);
        nq32 += __shfl_xor_sync(0xffffffffu, nq32, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (nq) atomicAdd(A.qcount, (unsigned long long) nq);
        if (nq32) atomicAdd(A.qcount32, (unsigned long long) nq32);
    }
}

// The classes without straight-line code (the largest f classes): a bra pair per
// warp, FP64. For each ket (bound order, all lanes) the lanes build the Hermite
// integrals R_tuv in per-warp shared tables, one order n of R^(n) at a time from
// the previous one's table (two tables in turn, so an order is one pass over its
// entries and one barrier), and then each lane contracts its bra components t:
// jp[t] += sum_u R_{t+u} D_u. A thread-per-pair kernel needs the whole table and
// the accumulators per thread (several KB), which overflow L1 for 128 threads per
// CTA. Bound by shared-memory accesses: an entry of the recursion reads its sources
// from a table of positions made once per CTA, and the integrals stand in rows of
// constant (t, u), so the contraction looks one row up per (u_x, u_y) and walks
// u_z at consecutive addresses. Decoding positions arithmetically for every entry
// and term, with a barrier per shell, made this kernel several times slower.
constexpr int kJWarpPairs = kJThreads / 32;   // bra pairs per CTA

// Position of (t, u, v), t + u + v <= L, with v fastest.
__host__ __device__ constexpr int row_pos(int L, int t, int u, int v)
{
    int p = 0;
    for (int i = 0; i < t; ++i) p += (L - i + 1) * (L - i + 2) / 2;
    for (int j = 0; j < u; ++j) p += L - t - j + 1;
    return p + v;
}

template <int LB, int LK>
struct JWarpShared {
    static constexpr int L = LB + LK, H = nherm_of(L);
    double boys[LSJK_BOYS_NBIN * 8];
    double R[kJWarpPairs][2][H];
    double dk[kJWarpPairs][nherm_of(LK)];
    ushort4 step[H];                            // (x: position, y, z: its sources, w: direction | factor << 2)
    unsigned short row[(L + 1) * (L + 1)];      // position of (t, u, 0)
    uint64_t mbar;
};

template <int LB, int LK>
__global__ void __launch_bounds__(kJThreads) k_coulomb_warp(JArgs A)
{
    constexpr int L = LB + LK, HB = nherm_of(LB), HK = nherm_of(LK), H = nherm_of(L), NT = (HB + 31) / 32;
    const int S = 4 + A.slots * HK;
    extern __shared__ __align__(128) unsigned char jwarp_smem[];
    JWarpShared<LB, LK>& sh = *reinterpret_cast<JWarpShared<LB, LK>*>(jwarp_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = *A.nbra, nk = *A.nket;
    const int g = blockIdx.z;   // the density (one per CTA z)
    const int ib = blockIdx.x * kJWarpPairs;
    const int j0 = blockIdx.y * A.chunk;
    if (ib >= nb || j0 >= nk) return;
    if (A.bbound[ib] * A.kbound[j0] < A.thresp) return;
    // the recursion's steps in shell order: R_tuv from its neighbours one and two below
    // in the first non-zero direction
    for (int k = threadIdx.x; k < H; k += kJThreads) {
        int N = 0;
        while (nherm_of(N) <= k) ++N;
        const int r = N ? k - nherm_of(N - 1) : 0;
        int ii = 0;
        while ((ii + 1) * (ii + 2) / 2 <= r) ++ii;
        const int t[3] = {N - ii, ii - (r - ii * (ii + 1) / 2), r - ii * (ii + 1) / 2};
        const int d = t[0] > 0 ? 0 : (t[1] > 0 ? 1 : 2);
        const int n = t[d];
        auto below = [&](int by) {
            return n < by ? 0 : row_pos(L, t[0] - (d == 0 ? by : 0), t[1] - (d == 1 ? by : 0), t[2] - (d == 2 ? by : 0));
        };
        sh.step[k] = make_ushort4((unsigned short) row_pos(L, t[0], t[1], t[2]), (unsigned short) below(1),
                                  (unsigned short) below(2), (unsigned short) (d | (n > 1 ? n - 1 : 0) << 2));
    }
    for (int k = threadIdx.x; k < (L + 1) * (L + 1); k += kJThreads) {
        const int t = k / (L + 1), u = k % (L + 1);
        sh.row[k] = (unsigned short) (t + u <= L ? row_pos(L, t, u, 0) : 0);
    }
    if (!stage_bulk(sh.boys, A.boys, sizeof(sh.boys), &sh.mbar, A.status)) return;   // (with CTA barriers)
    const int i = ib + warp;
    if (i >= nb) return;
    double* dks = sh.dk[warp];
    const double p = A.bgeom[4L * i], Px = A.bgeom[4L * i + 1], Py = A.bgeom[4L * i + 2], Pz = A.bgeom[4L * i + 3];
    const float Bi = A.bbound[i];
    // this lane's bra components t = lane + 32 k: their row of the row table, and t_z
    int trow[NT], tz[NT];
    double jp[NT];
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        const int t = lane + 32 * k < HB ? lane + 32 * k : 0;
        int N = 0;
        while (nherm_of(N) <= t) ++N;
        const int r = N ? t - nherm_of(N - 1) : 0;
        int ii = 0;
        while ((ii + 1) * (ii + 2) / 2 <= r) ++ii;
        tz[k] = r - ii * (ii + 1) / 2;
        trow[k] = (N - ii) * (L + 1) + ii - tz[k];
        jp[k] = 0.0;
    }
    long nq = 0;
    const int j1 = min(j0 + A.chunk, nk);
    for (int j = j0; j < j1; ++j) {
        if (Bi * A.kbound[j] < A.thresp) break;   // kets in bound order
        const double* r = A.krec + (long) j * S;
        for (int k = lane; k < HK; k += 32) dks[k] = r[4 + g * HK + k];
        const double q = r[0];
        const double X = Px - r[1], Y = Py - r[2], Z = Pz - r[3];
        const double R2 = X * X + Y * Y + Z * Z;
        const double rs = rsqrt(p + q);
        const double rho = p * q * (rs * rs);
        ++nq;
        for (int tm = 0; tm < A.nterm; ++tm) {
            const double om = A.omega[tm];
            double d2 = 1.0, f = A.alpha[tm] * rs;
            if (om != -1.0) {
                const double w2 = om * om;
                d2 = w2 / (rho + w2);
                f *= sqrt(d2);
            }
            const double rhoe = rho * d2;
            double F[L + 1];
            boys_eval<L, double>(rhoe * R2, sh.boys, F);
            double a[L + 1];
            const double m2r = -2.0 * rhoe;
            double pw = f;
#pragma unroll
            for (int n = 0; n <= L; ++n) {
                a[n] = pw * F[n];
                pw *= m2r;
            }
            // R^(n), n = L .. 0, all orders up to L - n
            if (lane == 0) sh.R[warp][L & 1][0] = a[L];
            __syncwarp();
#pragma unroll
            for (int n = L - 1; n >= 0; --n) {
                const double* src = sh.R[warp][(n + 1) & 1];
                double* dst = sh.R[warp][n & 1];
                if (lane == 0) dst[0] = a[n];
#pragma unroll 2
                for (int k = 1 + lane; k < nherm_of(L - n); k += 32) {
                    const ushort4 e = sh.step[k];
                    const int d = e.w & 3;
                    const double D = d == 0 ? X : (d == 1 ? Y : Z);
                    dst[e.x] = fma(D, src[e.y], (double) (e.w >> 2) * src[e.z]);
                }
                __syncwarp();
            }
            const double* Rb = sh.R[warp][0];
            double sv[NT];
#pragma unroll
            for (int k = 0; k < NT; ++k) sv[k] = jp[k];
#pragma unroll
            for (int ux = 0; ux <= LK; ++ux)
#pragma unroll
                for (int uy = 0; uy <= LK - ux; ++uy) {
                    int at[NT];
#pragma unroll
                    for (int k = 0; k < NT; ++k) at[k] = sh.row[trow[k] + ux * (L + 1) + uy] + tz[k];
#pragma unroll
                    for (int uz = 0; uz <= LK - ux - uy; ++uz) {
                        const double dv = dks[herm_pos(ux, uy, uz)];
#pragma unroll
                        for (int k = 0; k < NT; ++k) sv[k] = fma(Rb[at[k] + uz], dv, sv[k]);
                    }
                }
#pragma unroll
            for (int k = 0; k < NT; ++k) jp[k] = sv[k];
            __syncwarp();   // the tables are rebuilt for the next term or ket
        }
    }
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        const int t = lane + 32 * k;
        if (t < HB && jp[k] != 0.0) atomicAdd(&A.jbra[g * A.jbra_stride + (long) i * HB + t], jp[k]);
    }
    if (lane == 0 && nq) atomicAdd(A.qcount, (unsigned long long) nq);
}

template <int LB, int LK>
void launch_j(Context* ctx, const JArgs& A0, int nbra_full, int nket_full)
{
    if (nbra_full == 0 || nket_full == 0) return;
    if constexpr (JQ<LB, LK>::loop) {
        // classes without straight-line code: a bra pair per warp, FP64, a density per CTA z.
        // A CTA holds few pairs, so the default chunk, halved while there are fewer than
        // four CTAs per multiprocessor, stays larger than the thread-per-pair kernel's
        // (each CTA makes its tables first)
        JArgs A = A0;
        const long tiles = (nbra_full + kJWarpPairs - 1) / kJWarpPairs;
        if (!A.tuned)
            for (A.chunk = kJChunk; A.chunk > 16 && tiles * ((nket_full + A.chunk - 1) / A.chunk) < 4L * ctx->nsm;)
                A.chunk >>= 1;
        dim3 grid((unsigned) tiles, (nket_full + A.chunk - 1) / A.chunk, A.ng);
        auto kern = k_coulomb_warp<LB, LK>;
        constexpr size_t smem = sizeof(JWarpShared<LB, LK>);
        // the shared-memory opt-in is a per-device function attribute: set it once per device
        static std::atomic<unsigned long long> devices{0};
        const unsigned long long bit = 1ull << (ctx->device & 63);
        if (smem > 48 * 1024 && !(devices.load(std::memory_order_acquire) & bit)) {
            LSJK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
            devices.fetch_or(bit, std::memory_order_acq_rel);
        }
        kern<<<grid, kJThreads, smem, ctx->stream>>>(A);
        LSJK_CUDA(cudaGetLastError());
        ctx->stats.kernel_launches++;
        return;
    }
    const JArgs& A = A0;
    // one launch for all densities: CTA z takes NG of them over the same ket
    // records (NG = the class's batch when there are that many, else 1)
    constexpr int NGB = j_batch<LB>();
    const bool batched = NGB > 1 && A.ng >= NGB;
    const int NG = batched ? NGB : 1;
    dim3 grid((nbra_full + kJThreads - 1) / kJThreads, (nket_full + A.chunk - 1) / A.chunk, (A.ng + NG - 1) / NG);
    if (batched)
        k_coulomb<LB, LK, NGB><<<grid, kJThreads, 0, ctx->stream>>>(A);
    else
        k_coulomb<LB, LK, 1><<<grid, kJThreads, 0, ctx->stream>>>(A);
    LSJK_CUDA(cudaGetLastError());
    ctx->stats.kernel_launches++;
}


} // namespace lsjk
