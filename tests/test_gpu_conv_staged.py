"""The two-stage convection kernel (csrc/convection_staged.cu, stream mode
wherever a slice fits its planes) at the edges of its segment rule: the
shortest lines, lines of one cell more and less than whole groups, more lines
than segments of the shortest length allow, long thin slices, and a slice too
large for its planes (one thread per line instead); boundary types of both
sweeps, periodic L included, and L lines with different CFL sub-cycle counts.
Held to the contracted kernels' tolerance of 1e-12 for one step: of the
largest value, and for cells above 1e-6 of it, of the largest value their
stencils reach (five cells along either line; the boundary values drawn here
are up to a thousand times the cells beside them, and a face is rounded
relative to the largest value it takes)."""
import numpy as np
import pytest
from scipy.ndimage import maximum_filter

from verb4d_b200 import workload as W

from test_gpu_conv_stream import BCS, TOL, conv_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,R", [(11, 11), (12, 13), (13, 12), (48, 25), (24, 101), (25, 73),
                                 (11, 200), (90, 13), (60, 150)])
@pytest.mark.parametrize("pbc,rl,ru", [("periodic", "value", "value"),
                                       ("periodic", "periodic", "periodic"),
                                       ("deriv", "deriv", "value"), ("value", "value", "deriv")])
def test_shapes_and_boundaries(gpu, oracle_lib, P, R, pbc, rl, ru):
    wl = W.make_workload(W.GridSpec(P, R, 3, 2), seed=P + R, sources=True, losses=True)
    f = wl.fields
    f["VP"] = f["VP"] * 0.05  # few sub-steps at the largest sizes
    rng = np.random.default_rng(R)
    f["psd"] = f["psd"] * np.exp(0.05 * rng.standard_normal(f["psd"].shape))
    f["psd"][-1] = f["psd"][0]
    wl.bc_types.update(Pl=BCS[pbc], Pu=BCS[pbc], Rl=BCS[rl], Ru=BCS[ru])
    for name, kind in (("Pl", pbc), ("Pu", pbc), ("Rl", rl), ("Ru", ru)):
        if kind != "periodic":
            f[name] = rng.uniform(0.0, 0.05, f[name].shape)
    if P == 25:  # L spacing shrinking along MLT: lines with their own sub-cycles
        fac = 1.0 / (1.0 + 7.0 * np.arange(P) / (P - 1))
        f["Rg"] = f["Rg"][0, 0] + (f["Rg"] - f["Rg"][0, 0]) * fac[:, None, None, None]
    got, ref, ns = conv_step(wl, oracle_lib)
    assert np.array_equal(ns, W.convection_substeps(wl))
    scale = np.abs(ref).max()
    assert np.abs(got - ref).max() <= TOL * scale
    near = maximum_filter(np.abs(ref), size=(11, 11, 1, 1), mode="nearest")
    big = np.abs(ref) > 1e-6 * scale
    assert np.all((np.abs(got - ref) <= TOL * near)[big])
