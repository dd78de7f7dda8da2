"""The blocked banded LU of the local systems (csrc/local.cu) at the edges of
its variants: pivots, PSD and band factors equal the oracle's unblocked
xGBTF2/xGBTRS bit for bit.  V around the row counts where the panel takes
another warp (24, 56, 88 rows), the narrowest and widest band, unknown counts
that leave partial last panels; coefficients that are constant (rows tie in
the pivot search), independent draws (interchanges), and near 2^1000 (the
branch that keeps xGBTF2's skips)."""
import numpy as np
import pytest

from verb4d_b200 import workload as W

from test_gpu_step import load_ctx

pytestmark = pytest.mark.gpu


def set_coefficients(wl, kind):
    f = wl.fields
    if kind == "constant":
        f["DVV"][:], f["DKK"][:], f["DVK"][:] = 0.864, 0.864, 0.25
    elif kind == "huge":
        for n in ("DVV", "DKK", "DVK"):
            f[n] *= 1e299


@pytest.mark.parametrize("kind", ["drawn", "constant", "huge"])
@pytest.mark.parametrize("V,K", [(7, 3), (8, 5), (22, 4), (23, 7), (24, 3), (54, 4), (55, 3),
                                 (56, 5), (87, 3), (88, 4), (101, 5), (110, 3), (111, 3)])
def test_factor_matches_oracle(gpu, oracle_lib, V, K, kind):
    wl = W.make_workload(W.GridSpec(2, 2, V, K), seed=V + K, sources=True, losses=True)
    set_coefficients(wl, kind)
    f = wl.fields
    c = load_ctx(wl)
    psd0 = c.download()
    c.local(wl.dt, wl.sub_dt)
    c.sync()
    psd1, piv = c.download(), c.local_pivots()
    band = {pr: c.local_factor_lapack(*pr)[0] for pr in [(0, 0), (1, 1)]}
    c.close()
    n, ldab = V * K, 3 * (V + 1) + 1
    for p in range(2):
        for r in range(2):
            s2 = lambda a: a[p, r]  # noqa: E731
            lu, ip = np.zeros(ldab * n), np.zeros(n, np.int64)
            st, ref = oracle_lib.diffusion_2d(
                s2(psd0), s2(f["Vg"]), s2(f["Kg"]), f["Vl"][p, r], f["Vu"][p, r], f["Kl"][p, r],
                f["Ku"][p, r], (1, 1, 2, 2), s2(f["DVV"]), s2(f["DKK"]), s2(f["DVK"]),
                s2(f["DVK"]), s2(f["G_local"]), s2(f["S"]), s2(f["loss_local"]), wl.dt, wl.sub_dt,
                lu=lu, ipiv=ip)
            assert st == 0
            assert np.array_equal(piv[p, r], ip)
            assert np.array_equal(psd1[p, r], ref, equal_nan=True)
            if (p, r) in band:
                got = band[p, r].reshape(n, ldab)
                for j in range(n):  # the rows of column j inside the matrix
                    lo = max(0, 2 * (V + 1) - j)
                    hi = min(ldab, 2 * (V + 1) + n - j)
                    assert np.array_equal(got[j, lo:hi], lu.reshape(n, ldab)[j, lo:hi],
                                          equal_nan=True), (p, r, j)
