"""Zeros of both signs through the exact two-stage convection: the same bits as
the oracle, the signs of zeros included (a cell that takes no source term has
nothing added to it, and a line that waits for others is carried over as it
is).  Shapes of the 2-, 5- and 8-cell segments; without convection losses
(exp() may differ in the last bit from the host's)."""
import numpy as np
import pytest

import oracle as O
from verb4d_b200 import workload as W

from test_gpu_conv_stream import BCS
from test_gpu_step import load_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,R", [(12, 13), (17, 19), (24, 25), (24, 51), (36, 50)])
@pytest.mark.parametrize("pbc,rbc", [("periodic", "value"), ("periodic", "periodic"),
                                     ("value", "value"), ("deriv", "deriv")])
def test_signs_of_zeros(gpu, oracle_lib, P, R, pbc, rbc):
    wl = W.make_workload(W.GridSpec(P, R, 20, 16), seed=P, sources=True)
    f = wl.fields
    rng = np.random.default_rng(R)
    f["VP"] = f["VP"] * 0.02
    f["psd"] = np.where(rng.uniform(size=f["psd"].shape) < 0.9, -0.0, f["psd"])
    f["psd"][:, :, 1::2] = -0.0  # whole slices of zeros
    f["psd"][-1] = f["psd"][0]
    f["S"] = np.where(rng.uniform(size=f["S"].shape) < 0.5, -0.0, 0.0)
    for n in ("Pl", "Pu", "Rl", "Ru"):
        f[n] = np.where(rng.uniform(size=f[n].shape) < 0.5, -0.0, 0.0)
    if P == 24:  # L spacing shrinking along MLT: lines with their own sub-cycles
        fac = 1.0 / (1.0 + 3.0 * np.arange(P) / (P - 1))
        f["Rg"] = f["Rg"][0, 0] + (f["Rg"] - f["Rg"][0, 0]) * fac[:, None, None, None]
    wl.bc_types.update(Pl=BCS[pbc], Pu=BCS[pbc], Rl=BCS[rbc], Ru=BCS[rbc])
    flags = dict(wl.flags, run_convection=1, run_radial=0, run_local=0)
    st = O.OracleStepper(dict(W.oracle_inputs(wl), flags=flags), oracle_lib)
    st.step(wl.dt, wl.sub_dt, True)
    c = load_ctx(wl)
    c.convection(wl.dt)
    c.sync()
    got = c.download()
    c.close()
    assert np.signbit(st.psd[st.psd == 0.0]).any()
    assert np.array_equal(got.view(np.int64), st.psd.view(np.int64))
