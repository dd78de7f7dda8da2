"""The exact form of the two-stage convection kernel: bit-identical to the
oracle over the launch rule's shapes (2-, 5- and 8-cell segments, up to 512
threads, lines it leaves to the line-job kernel), boundary types, mixed
directions along a line, G other than 1, cells of zero and of magnitudes whose
quotients leave the normal range (infinities and NaN follow, at the same cells),
and per-line CFL sub-cycles.  Without
convection loss rates (exp() may differ in the last bit from the host's)."""
import numpy as np
import pytest

import oracle as O
from verb4d_b200 import workload as W

from test_gpu_conv_stream import BCS
from test_gpu_step import load_ctx

pytestmark = pytest.mark.gpu


def workload(P, R, pbc="periodic", rl="value", ru="value"):
    wl = W.make_workload(W.GridSpec(P, R, 3, 2), seed=P + R, sources=True)
    f = wl.fields
    f["VP"] = f["VP"] * 0.05
    rng = np.random.default_rng(R)
    f["psd"] = f["psd"] * np.exp(0.05 * rng.standard_normal(f["psd"].shape))
    f["psd"][-1] = f["psd"][0]
    wl.bc_types.update(Pl=BCS[pbc], Pu=BCS[pbc], Rl=BCS[rl], Ru=BCS[ru])
    for name, kind in (("Pl", pbc), ("Pu", pbc), ("Rl", rl), ("Ru", ru)):
        if kind != "periodic":
            f[name] = rng.uniform(0.0, 0.05, f[name].shape)
    return wl, rng


def check(wl, oracle_lib):
    flags = dict(wl.flags, run_convection=1, run_radial=0, run_local=0)
    st = O.OracleStepper(dict(W.oracle_inputs(wl), flags=flags), oracle_lib)
    st.step(wl.dt, wl.sub_dt, True)
    c = load_ctx(wl)
    c.convection(wl.dt)
    c.sync()
    got, ns = c.download(), c.convection_substeps()
    c.close()
    assert np.array_equal(ns, W.convection_substeps(wl))
    assert np.array_equal(got, st.psd, equal_nan=True)


@pytest.mark.parametrize("P,R", [(11, 11), (12, 13), (13, 40), (24, 25), (13, 90), (24, 51), (36, 50),
                                 (48, 101), (90, 13), (60, 150), (11, 512)])
@pytest.mark.parametrize("pbc,rl,ru", [("periodic", "value", "value"), ("deriv", "deriv", "value"),
                                       ("value", "periodic", "periodic")])
def test_shapes(gpu, oracle_lib, P, R, pbc, rl, ru):
    check(workload(P, R, pbc, rl, ru)[0], oracle_lib)


@pytest.mark.parametrize("kind", ["mixed", "jacobian", "range", "subcycles"])
def test_inputs(gpu, oracle_lib, kind):
    wl, rng = workload(25, 40)
    f = wl.fields
    if kind == "mixed":        # directions that change from face to face, and zero velocities
        f["VP"] = f["VP"] * rng.choice([-1.0, 0.0, 1.0], f["VP"].shape)
        f["VR"] = f["VR"] * rng.choice([-1.0, 0.0, 1.0], f["VR"].shape)
    elif kind == "jacobian":
        f["G_conv"] = rng.uniform(0.1, 9.0, f["G_conv"].shape)
    elif kind == "range":
        f["psd"] = f["psd"] * 10.0 ** rng.integers(-300, 2, f["psd"].shape)
        f["psd"][rng.uniform(size=f["psd"].shape) < 0.3] = 0.0
        f["psd"][-1] = f["psd"][0]
        f["G_conv"] = 10.0 ** rng.uniform(-140, 140, f["G_conv"].shape)
    else:
        fac = 1.0 / (1.0 + 7.0 * np.arange(25) / 24)
        f["Rg"] = f["Rg"][0, 0] + (f["Rg"] - f["Rg"][0, 0]) * fac[:, None, None, None]
    check(wl, oracle_lib)
