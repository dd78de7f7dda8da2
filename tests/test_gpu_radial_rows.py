"""The radial pass at the edges of its row chunks (three rows where it
factorises, eight where it solves with the cached recurrence): the smallest
lines, every remainder of both chunk lengths, both boundary types at both ends,
a step that factorises followed by one that does not, sources, and lines whose
geometry factors leave the range of the shared reciprocals (quotients divided
one by one).  Bit for bit against the oracle."""
import numpy as np
import pytest

from verb4d_b200 import Context
from verb4d_b200 import workload as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types", [(1, 1), (2, 1), (1, 2), (2, 2)])
@pytest.mark.parametrize("R", [3, 4, 5, 6, 8, 9, 10, 11, 17, 27])
def test_radial_rows(gpu, oracle_lib, R, types):
    spec = W.GridSpec(3, R, 5, 9)   # 135 lines: a block and a ragged one
    wl = W.make_workload(spec, seed=R, sources=True, losses=True)
    f = wl.fields
    f["G_radial"][0, :, 1, 2] *= 2.0 ** 500
    f["G_radial"][1, :, 2, 3] *= 2.0 ** -500
    f["psd"][2, :, 3, 4] *= 2.0 ** -600
    f["DLL"][0, :, 0, 0] = 0.0
    c = Context(*spec.shape)
    c.set_bc_types(dict(wl.bc_types, Ll=types[0], Lu=types[1]))
    c.set_options(1, 0, 1, 0)
    for k in ("psd", "Lg", "DLL", "G_radial", "S", "loss_radial", "Ll", "Lu"):
        c.upload(k, f[k])
    want = f["psd"].copy()
    for dt in (wl.dt, wl.dt, 0.5 * wl.dt):
        c.radial(dt)
        c.sync()
        for p in range(3):
            for v in range(5):
                for k in range(9):
                    ln = lambda a: a[p, :, v, k]  # noqa: E731
                    st, want[p, :, v, k] = oracle_lib.diffusion_1d(
                        ln(want), ln(f["Lg"]), f["Ll"][p, v, k], f["Lu"][p, v, k], *types,
                        ln(f["DLL"]), ln(f["G_radial"]), ln(f["S"]), ln(f["loss_radial"]), dt)
                    assert st == 0
        assert np.array_equal(c.download(), want, equal_nan=True)
    assert np.isfinite(want[0, :, 2]).all()
    c.close()
