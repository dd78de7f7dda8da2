"""The contracted two-stage convection (stream mode) beside a value that is not
finite, or beside which its neighbours vanish.  Its regrouped polynomial leaves
out one end of the stencil, and its differences of infinities cancel, so slices
that hold such values take the reference's sums in a second launch.

Every slice carries a monotone, convex profile along MLT (all limiters decide
clearly: the contracted form may round their comparisons differently) with one
NaN, infinity or 1e300 at one of its cells, in either direction of transport.
Not finite at the oracle's cells; elsewhere within the contracted kernels' 1e-12
of the profile.  Slices without such a value stand among them."""
import numpy as np
import pytest

import oracle as O
from verb4d_b200 import workload as W

from test_gpu_conv_stream import BCS, TOL
from test_gpu_step import load_ctx

pytestmark = pytest.mark.gpu

VALUES = (np.nan, np.inf, -np.inf, 1e300, None)


@pytest.mark.parametrize("bc", ["value", "periodic"])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("P,R", [(11, 11), (13, 12), (24, 25), (60, 13), (48, 101)])
def test_one_value(gpu, oracle_lib, P, R, sign, bc):
    wl = W.make_workload(W.GridSpec(P, R, P, len(VALUES)), seed=P)
    f = wl.fields
    shape = f["psd"].shape
    profile = np.exp(0.1 * np.arange(P))[:, None, None, None] * np.ones(shape)
    f["psd"] = profile.copy()
    for m in range(P):
        for k, v in enumerate(VALUES):
            if v is not None:
                f["psd"][m, :, m, k] = v
    dx = f["Pg"][1, 0, 0, 0] - f["Pg"][0, 0, 0, 0]
    f["VP"] = np.full(shape, sign * 0.2 * dx / wl.dt)  # Courant number 0.2: one sub-step
    f["VR"] = np.zeros(shape)
    f["G_conv"], f["S"], f["loss_conv"] = np.ones(shape), np.zeros(shape), np.zeros(shape)
    wl.bc_types.update(Pl=BCS[bc], Pu=BCS[bc], Rl=BCS["value"], Ru=BCS["value"])
    if bc == "value":
        f["Pl"], f["Pu"] = np.full(f["Pl"].shape, 1.0), np.full(f["Pu"].shape, np.exp(0.1 * (P - 1)))
    f["Rl"], f["Ru"] = f["psd"][:, 0].copy(), f["psd"][:, -1].copy()
    flags = dict(wl.flags, run_convection=1, run_radial=0, run_local=0)
    st = O.OracleStepper(dict(W.oracle_inputs(wl), flags=flags), oracle_lib)
    with np.errstate(all="ignore"):
        st.step(wl.dt, wl.sub_dt, True)
    c = load_ctx(wl)
    c.set_convection_arith("stream")
    assert c.convection_kernel() == "staged"
    c.convection(wl.dt)
    c.sync()
    got = c.download()
    c.close()
    finite = np.isfinite(st.psd) & (np.abs(st.psd) < 1e200)
    assert np.array_equal(np.isfinite(got) & (np.abs(got) < 1e200), finite)
    assert finite[:, :, :, :4].any() and not finite[:, :, :, :4].all()
    assert np.abs(got[finite] - st.psd[finite]).max() <= TOL * profile.max()
