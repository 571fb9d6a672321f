"""The FP32 K pass's asymptotic Rys rule, carried in pairs of floats (lsjk_device.cuh:
rys_asym_pairs), compiled for the CPU as it stands: its roots and weights against 80-bit
arithmetic, beside the FP64 evaluation rounded to FP32, from the last table bin upward, for
every error the hardware's reciprocal square root may have (2 ulp)."""
import ctypes
import os
import re

import numpy as np
import pytest

from host_code import CSRC, CUDA_WORDS, compile_host, source_part

CODE = """
#include <cmath>
#include <limits>
static int ulps;
static float rsqrtf(float x)
{
    float r = (float) (1.0L / sqrtl((long double) x));
    for (int k = 0; k < (ulps < 0 ? -ulps : ulps); ++k) r = nextafterf(r, ulps < 0 ? 0.0f : 1e30f);
    return r;
}
#include "tables/quad_tables.inc"
%s
template <int N>
static void run_n(long n, const float* rho, const float* d2, const float* RR, double* out)
{
    for (long k = 0; k < n; ++k) {
        float t2[N], w[N];
        rys_asym_pairs<N>(rho[k], d2[k], RR[k], t2, w);
        const long double T = (long double) rho[k] * d2[k] * RR[k], R = 1.0L / sqrtl(T);
        const double r = 1.0 / sqrt((double) rho[k] * (double) d2[k] * (double) RR[k]);
        for (int i = 0; i < N; ++i) {
            const double s = kRysAsymT[N * LSJK_RYS_NMAX + i], h = kRysAsymW[N * LSJK_RYS_NMAX + i];
            const double t = s * r;
            const float want[2] = {(float) (t * t), (float) (h * r)}, got[2] = {t2[i], w[i]};
            const long double exact[2] = {s * (long double) s / T, h * R};
            for (int q = 0; q < 2; ++q) {
                const double a = fabsl(got[q] / exact[q] - 1.0L), b = fabsl(want[q] / exact[q] - 1.0L);
                out[0] = fmax(out[0], a);
                out[1] = fmax(out[1], b);
                out[2] += a * a;
                out[3] += b * b;
                out[4] += got[q] != want[q];
                out[5] += 1.0;
            }
        }
    }
}
extern "C" void run(int N, int err, long n, const float* rho, const float* d2, const float* RR, double* out)
{
    ulps = err;
    switch (N) {
    case 1: run_n<1>(n, rho, d2, RR, out); break;
    case 2: run_n<2>(n, rho, d2, RR, out); break;
    case 3: run_n<3>(n, rho, d2, RR, out); break;
    case 4: run_n<4>(n, rho, d2, RR, out); break;
    case 5: run_n<5>(n, rho, d2, RR, out); break;
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not os.path.exists(os.path.join(CSRC, "tables", "quad_tables.inc")):
        pytest.skip("quadrature tables not generated (run the build)")
    part = source_part("lsjk_device.cuh", "// The asymptotic Rys nodes as pairs of floats", "// Root i alone of the N-point rule")
    return compile_host(tmp_path_factory.mktemp("rys"), CUDA_WORDS + CODE % part)


# the rules of the FP32 classes: (ss|ss) to (dd|dd)
@pytest.mark.parametrize("N", [1, 2, 3, 4, 5])
def test_as_exact_as_fp64_rounded(lib, N):
    inc = open(os.path.join(CSRC, "tables", "quad_tables.inc")).read()
    row = lambda name: [float(v) for v in re.search(r"%s\[\d+\] = \{(.*?)\};" % name, inc).group(1).split(",")]
    first = row("kRysTmax")[N] * (1.0 - 1.0 / row("kRysNbin")[N])
    rng = np.random.default_rng(N)
    n = 100000
    rho = np.exp(rng.uniform(np.log(1e-3), np.log(1e5), n)).astype(np.float32)
    d2 = np.where(rng.random(n) < 0.5, 1.0, np.exp(rng.uniform(np.log(1e-5), 0.0, n))).astype(np.float32)
    T = first * np.exp(rng.uniform(0.0, np.log(1e8), n) * rng.random(n))
    RR = (T / (rho.astype(np.float64) * d2)).astype(np.float32)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    out = np.zeros(6)
    for err in (-2, -1, 0, 1, 2):
        lib.run(N, err, ctypes.c_long(n), ptr(rho), ptr(d2), ptr(RR), ptr(out))
    print("N = %d: largest %.9e (FP64 rounded %.9e), rms %.6e (%.6e), %d of %d round differently"
          % (N, out[0], out[1], (out[2] / out[5]) ** 0.5, (out[3] / out[5]) ** 0.5, out[4], out[5]))
    # half an ulp of FP32 is 2^-24; the pairs are off by a few 2^-47, so about 2^-20 of the samples
    # lie close enough to a rounding boundary to go the other way (four times that allowed)
    assert out[0] <= 2.0 ** -24 * (1.0 + 1e-5)
    assert out[0] <= out[1] * (1.0 + 1e-6)
    assert abs(out[2] / out[3] - 1.0) < 1e-6
    assert out[4] <= 4e-6 * out[5]
