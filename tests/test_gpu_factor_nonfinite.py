"""The panel factorisation where the matrix holds NaN, infinities or pivots that
are exactly zero: the oracle's pivots and factors bit for bit (NaN at the same
places) and its status.  xGBTF2 updates every row that a pivot reaches, rows
of zero multipliers included (an infinite u makes them NaN), and no other;
interchanges in a panel move rows across that border."""
import numpy as np
import pytest

from verb4d_b200 import VerbError
from verb4d_b200 import workload as W

from test_gpu_step import load_ctx

pytestmark = pytest.mark.gpu


def spoil(wl, kind, rng):
    f = wl.fields
    names = ("DVV", "DKK", "DVK")
    if kind == "interchanges":
        for n in names:
            f[n] = rng.uniform(-1, 1, f[n].shape) * 10.0 ** rng.uniform(-3, 3, f[n].shape)
    elif kind in ("nan", "inf", "both"):
        for n in names:
            f[n] = rng.uniform(-1, 1, f[n].shape) * 10.0 ** rng.uniform(-3, 3, f[n].shape)
        v = f[rng.choice(names)].reshape(-1)
        idx = rng.integers(0, v.size, 4)
        v[idx] = {"nan": [np.nan] * 4, "inf": [np.inf, -np.inf] * 2,
                  "both": [np.nan, np.inf, np.nan, -np.inf]}[kind]
    elif kind == "jacobian":
        v = f["G_local"].reshape(-1)
        v[rng.integers(0, v.size, 3)] = (np.inf, np.nan, 1e-310)
    elif kind == "overflow":     # drawn coefficients, most of them infinite
        for n in names:
            f[n] = f[n] * rng.choice([1e300, 1e308, 1e310], f[n].shape)
    elif kind == "zero":         # whole rows of zeros: pivots that are zero
        f["loss_local"][:] = 1.0 / wl.sub_dt
        for n in names:
            f[n][:] = 0.0


@pytest.mark.parametrize("kind", ["interchanges", "nan", "inf", "both", "jacobian", "overflow", "zero"])
@pytest.mark.parametrize("V,K", [(7, 5), (8, 7), (9, 13), (16, 11), (23, 6), (24, 9), (31, 8), (55, 5),
                                 (56, 7), (88, 4), (100, 6), (111, 4)])
def test_nonfinite(gpu, oracle_lib, V, K, kind):
    rng = np.random.default_rng([V, K, len(kind)])
    wl = W.make_workload(W.GridSpec(2, 3, V, K), seed=V + K, sources=True, losses=True)
    with np.errstate(over="ignore", invalid="ignore"):
        spoil(wl, kind, rng)
    f = wl.fields
    c = load_ctx(wl)
    psd0 = c.download()
    failed = False
    try:
        c.local(wl.dt, wl.sub_dt)
        c.sync()
    except VerbError as e:
        assert e.status == 1  # VERB_ERR_PIVOT
        failed = True
    piv = c.local_pivots()
    n, ldab = V * K, 3 * (V + 1) + 1
    status = []
    for p in range(2):
        for r in range(3):
            s2 = lambda a: a[p, r]  # noqa: E731
            lu, ip = np.zeros(ldab * n), np.zeros(n, np.int64)
            with np.errstate(all="ignore"):
                st, _ = oracle_lib.diffusion_2d(
                    s2(psd0), s2(f["Vg"]), s2(f["Kg"]), f["Vl"][p, r], f["Vu"][p, r], f["Kl"][p, r],
                    f["Ku"][p, r], (1, 1, 2, 2), s2(f["DVV"]), s2(f["DKK"]), s2(f["DVK"]),
                    s2(f["DVK"]), s2(f["G_local"]), s2(f["S"]), s2(f["loss_local"]), wl.dt, wl.sub_dt,
                    lu=lu, ipiv=ip)
            status.append(st)
            assert np.array_equal(piv[p, r], ip), (p, r)
            got = c.local_factor_lapack(p, r)[0].reshape(n, ldab)
            want = lu.reshape(n, ldab)
            for j in range(n):  # the rows of column j inside the matrix
                lo, hi = max(0, 2 * (V + 1) - j), min(ldab, 2 * (V + 1) + n - j)
                assert np.array_equal(got[j, lo:hi], want[j, lo:hi], equal_nan=True), (p, r, j)
    c.close()
    assert failed == any(status)
