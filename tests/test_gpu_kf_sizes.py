"""The radial and the (MLT, L) filters at the edges of their matrix-product
kernels: sizes that fill no 8-row tile, T in shared memory or (R > 112) in the
workspace, odd and even state counts (8- and 16-byte copies), the smallest
grids, every point observed and columns without observations.  Radial columns
against the oracle at the tolerance of tests/test_gpu_kf.py, slices of the
(MLT, L) filter against the restatement at that of tests/test_gpu_kfconv.py."""
import numpy as np
import pytest

from verb4d_b200 import Context
from verb4d_b200 import workload as W

from test_gpu_kf import KF_RTOL
from test_gpu_kfconv import ME, OE, TOL, make_obs, oracle_slice, rel
from test_gpu_step import load_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [3, 7, 8, 9, 33, 112, 113, 128])
def test_radial_sizes(gpu, oracle_lib, R):
    spec = W.GridSpec(2, R, 3, 2)
    wl = W.make_workload(spec, seed=R)
    f = wl.fields
    rng = np.random.default_rng(R)
    obs = np.full(spec.shape, np.nan)
    if R > 3:
        seen = rng.uniform(size=spec.shape) < 0.2
        seen[:, :, 0, 0] = True   # every point of a column
    else:
        seen = np.ones(spec.shape, bool)
    seen[:, :, 2, 1] = False      # none
    seen[:, 0] = seen[:, -1] = False
    obs[seen] = f["psd"][seen] * np.exp(0.05 * rng.standard_normal(int(seen.sum())))
    c = Context(*spec.shape)
    c.set_bc_types(wl.bc_types)
    for k in ("psd", "Rg", "DLL", "G_radial", "Ll", "Lu"):
        c.upload(k, f[k])
    me, oe = 1e-4, 1e-3
    outs = []
    for _ in range(2):
        c.assimilate_radial(obs, wl.dt, me, oe, p_index=1)
        c.sync()
        outs.append(c.download())
    c.close()
    assert np.array_equal(outs[1][0], f["psd"][0])  # the other MLT is left alone
    for v in range(3):
        for k in range(2):
            ln = lambda a: np.ascontiguousarray(a[1, :, v, k])  # noqa: E731
            x, pa = ln(f["psd"]), np.zeros((R, R))
            for u in range(2):
                st, x, pa, *_ = oracle_lib.kf_diffusion_1d(
                    x, pa, ln(f["Rg"]), ln(f["DLL"]), ln(f["G_radial"]), float(f["Ll"][1, v, k]),
                    float(f["Lu"][1, v, k]), 1, 1, ln(obs), wl.dt, me, oe)
                assert st == 0
                assert rel(outs[u][1, :, v, k], x) < KF_RTOL, (v, k, u)


@pytest.mark.parametrize("P,R", [(3, 3), (5, 13), (8, 8), (9, 15), (11, 11)])
def test_convection_filter_sizes(gpu, P, R):
    wl = W.make_workload(W.GridSpec(P, R, 2, 2), seed=P * R, sources=True)
    obs = make_obs(wl, 7, 0.2)
    c = load_ctx(wl)
    c.assimilate_convection(obs, wl.dt, ME, OE, use_log=True, has_vx_updated=True, slice_chunk=3)
    for v in range(2):
        for k in range(2):
            x, pa, mm = oracle_slice(wl, wl.fields["psd"], np.zeros((P * R, P * R)), None, obs, v, k,
                                     True, True)
            gpa, gm = c.convection_da_state(v, k)
            assert rel(gm, mm) < 1e-12
            assert rel(gpa, pa) < TOL
            assert rel(c.download()[:, :, v, k], x) < TOL
    c.close()
