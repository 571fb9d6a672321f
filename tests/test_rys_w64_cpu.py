"""The FP64 kernels' Rys weight tables (w itself, ten coefficients per bin) against the
generator's Golub-Welsch rule, evaluated as the device does: bin edges, both ends of
the range and random points, for the rules the kernels use (up to (ff|ff) and its gradient)."""
import importlib.util
import os
import re

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INC = os.path.join(ROOT, "lightspeed_b200", "csrc", "tables", "quad_tables.inc")


@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7])
def test_fp64_weight_tables(n):
    if not os.path.exists(INC):
        pytest.skip("quadrature tables not generated (run the build)")
    spec = importlib.util.spec_from_file_location("gen_tables", os.path.join(ROOT, "lightspeed_b200", "tables",
                                                                            "gen_tables.py"))
    gen = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(gen)
    txt = open(INC).read()

    def arr(name):
        return np.array([float(v) for v in re.search(r"%s\[\d+\] = \{(.*?)\};" % name, txt, re.S).group(1).split(",")])

    nbin, tmax = arr("kRysNbin").astype(int), arr("kRysTmax")
    nc = gen.NCOEF_W64
    start = sum(m * nbin[m] * nc for m in range(2, n))
    w64 = arr("kRysW64")[start:start + n * nbin[n] * nc].reshape(n, nbin[n], nc)
    edges = np.arange(nbin[n]) * (tmax[n] / nbin[n])
    T = np.unique(np.concatenate([[0.0, 1e-9], edges[::7], edges[::7] + 1e-10, [tmax[n] * (1 - 1e-12)],
                                  np.random.default_rng(n).uniform(0.0, tmax[n], 60)]))
    for t in T:
        u = t * (nbin[n] / tmax[n])
        b = min(int(u), nbin[n] - 1)
        x = 2.0 * (u - b) - 1.0
        w = w64[:, b, nc - 1]
        for k in range(nc - 2, -1, -1):
            w = w * x + w64[:, b, k]
        # interpolation error below 1e-15; the generator's own rule is good to ~1e-14
        assert np.max(np.abs(w / gen.rys_exact(n, t)[1] - 1.0)) < 5e-14
