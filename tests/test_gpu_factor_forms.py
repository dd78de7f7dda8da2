"""The factorisation of the local systems by panels with FP32 factors, and over
older factors, at the edges of its variants (V = 15 | 16, where FP32 columns begin to
hold a parked row, 8 likewise in FP64, and 23 | 24, 55 | 56, 87 | 88, where the panel
takes another warp).

FP32 factors are the FP64 ones rounded: without refinement the solution equals,
bit for bit, the oracle's solve with its own factors rounded to FP32.  A
context that factorises coefficients with many interchanges, then others (every
entry of the old factors must be written again), gives the bits of a fresh
context, in both precisions and both orders."""
import numpy as np
import pytest

from verb4d_b200 import workload as W

from test_gpu_factor import set_coefficients
from test_gpu_step import load_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["drawn", "constant"])
@pytest.mark.parametrize("V,K", [(7, 5), (8, 5), (15, 4), (16, 5), (22, 3), (23, 4), (24, 5), (54, 3),
                                 (55, 4), (56, 3), (87, 3), (88, 4), (111, 3)])
def test_fp32_factors(gpu, oracle_lib, V, K, kind):
    wl = W.make_workload(W.GridSpec(2, 2, V, K), seed=V + K, sources=True, losses=True)
    set_coefficients(wl, kind)
    f = wl.fields
    c = load_ctx(wl)
    c.set_local_precision("mixed", 0)
    psd0 = c.download()
    c.local(wl.dt, wl.sub_dt)
    c.sync()
    psd1, piv = c.download(), c.local_pivots()
    c.close()
    n, ldab = V * K, 3 * (V + 1) + 1
    for p in range(2):
        for r in range(2):
            s2 = lambda a: a[p, r]  # noqa: E731
            args = (s2(psd0), s2(f["Vg"]), s2(f["Kg"]), f["Vl"][p, r], f["Vu"][p, r], f["Kl"][p, r],
                    f["Ku"][p, r], (1, 1, 2, 2), s2(f["DVV"]), s2(f["DKK"]), s2(f["DVK"]),
                    s2(f["DVK"]), s2(f["G_local"]), s2(f["S"]), s2(f["loss_local"]), wl.dt, wl.sub_dt)
            lu, ip = np.zeros(ldab * n), np.zeros(n, np.int64)
            st, _ = oracle_lib.diffusion_2d(*args, lu=lu, ipiv=ip)
            assert st == 0
            assert np.array_equal(piv[p, r], ip)
            lu32 = lu.astype(np.float32).astype(np.float64)
            st, want = oracle_lib.diffusion_2d(*args, lu=lu32, ipiv=ip, recompute=False)
            assert st == 0
            assert np.array_equal(psd1[p, r], want, equal_nan=True)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("V,K", [(7, 9), (8, 9), (15, 7), (16, 7), (23, 6), (24, 6), (56, 4), (88, 3),
                                 (101, 4), (111, 3)])
def test_over_older_factors(gpu, V, K, prec):
    kinds = ("drawn", "constant", "huge", "drawn")
    wls = []
    for i, kind in enumerate(kinds):
        wl = W.make_workload(W.GridSpec(2, 3, V, K), seed=V + K + i, sources=True, losses=True)
        set_coefficients(wl, kind)
        wls.append(wl)
    want = []
    for wl in wls:
        c = load_ctx(wl)
        c.set_local_precision(prec, 0)
        c.local(wl.dt, wl.sub_dt)
        c.sync()
        want.append((c.download(), c.local_pivots()))
        c.close()
    c = load_ctx(wls[0])
    c.set_local_precision(prec, 0)
    for wl, (psd, piv) in zip(wls, want):
        for k in ("psd", "Vg", "Kg", "DVV", "DKK", "DVK", "G_local", "S", "loss_local", "Vl", "Vu",
                  "Kl", "Ku"):
            c.upload(k, wl.fields[k])
        c.local(wl.dt, wl.sub_dt)
        c.sync()
        assert np.array_equal(c.local_pivots(), piv)
        assert np.array_equal(c.download(), psd, equal_nan=True)
    c.close()
