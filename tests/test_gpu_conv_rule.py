"""The exact convection's choice of kernel and segments: the line-job kernel
where its sub-step is the shorter one (short lines; the two-stage kernel took
up to 17 % longer there), the two-stage kernel elsewhere; and both sides of the
rules on points and slices bit for bit against the oracle: 2-cell segments for
few slices (up to 512 threads), 5- and 8-cell ones for more, with every
boundary type and with directions that change from face to face."""
import numpy as np
import pytest

from verb4d_b200 import Context
from verb4d_b200 import workload as W

from test_gpu_conv_staged_exact import check
from test_gpu_conv_stream import BCS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,kernel", [
    ((12, 13, 31, 31), "lines"), ((16, 16, 31, 31), "lines"), ((22, 19, 31, 31), "lines"),
    ((23, 32, 31, 20), "lines"), ((22, 27, 31, 31), "lines"), ((20, 24, 45, 30), "lines"),
    ((12, 20, 31, 31), "staged"), ((19, 20, 31, 20), "staged"), ((24, 25, 31, 31), "staged"),
    ((26, 26, 31, 20), "staged"), ((23, 32, 19, 17), "staged"), ((22, 19, 19, 17), "staged"),
    ((24, 51, 31, 31), "staged"), ((48, 101, 31, 31), "staged"), ((12, 13, 61, 61), "staged"),
    ((24, 25, 61, 61), "staged"), ((24, 51, 61, 61), "lines"), ((48, 101, 61, 61), "lines")])
def test_kernel(gpu, shape, kernel):
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the counts are for 148 SMs")
    c = Context(*shape)
    assert c.convection_kernel() == kernel
    c.close()


@pytest.mark.parametrize("P,R,V,K", [(22, 27, 10, 2), (24, 42, 10, 3), (36, 28, 37, 10), (13, 75, 3, 2),
                                     (23, 32, 31, 12), (24, 25, 24, 20), (26, 26, 24, 16),
                                     (24, 42, 24, 16), (24, 51, 20, 19), (36, 50, 20, 19)])
@pytest.mark.parametrize("pbc,rl,ru", [("periodic", "value", "value"), ("deriv", "deriv", "value"),
                                       ("value", "periodic", "periodic")])
def test_both_sides(gpu, oracle_lib, P, R, V, K, pbc, rl, ru):
    wl = W.make_workload(W.GridSpec(P, R, V, K), seed=P + R, sources=True)
    f = wl.fields
    rng = np.random.default_rng(R)
    f["VP"] = f["VP"] * 0.01 * rng.choice([-1.0, 1.0], f["VP"].shape)
    f["VR"] = f["VR"] * rng.choice([-1.0, 0.0, 1.0], f["VR"].shape)
    f["psd"] = f["psd"] * np.exp(0.05 * rng.standard_normal(f["psd"].shape))
    f["psd"][-1] = f["psd"][0]
    wl.bc_types.update(Pl=BCS[pbc], Pu=BCS[pbc], Rl=BCS[rl], Ru=BCS[ru])
    for name, kind in (("Pl", pbc), ("Pu", pbc), ("Rl", rl), ("Ru", ru)):
        if kind != "periodic":
            f[name] = rng.uniform(0.0, 0.05, f[name].shape)
    check(wl, oracle_lib)
