"""Slices at the shared-memory limit of the convection kernels: the largest whose
planes fit the two-stage kernel, those a few bytes beyond (its static part
counts), and the next.  Every one runs, in the exact form bit for bit and in
the contracted one at 1e-12 of the largest value.  Slices a few bytes beyond
the line-job kernels' own limit, which no kernel holds, are refused as such."""
import numpy as np
import pytest

import oracle as O
from verb4d_b200 import VerbError
from verb4d_b200 import workload as W

from test_gpu_step import load_ctx

pytestmark = pytest.mark.gpu
TOL = 1e-12  # contracted kernels, one step (tests/test_gpu_conv_stream.py)


def slice_workload(P, R):
    wl = W.make_workload(W.GridSpec(P, R, 2, 1), seed=R, sources=True)
    wl.fields["VP"] = wl.fields["VP"] * (0.3 / P)  # few sub-steps
    return wl


@pytest.mark.parametrize("P,R", [(33, 199), (33, 200), (33, 201), (33, 202), (319, 17), (319, 18),
                                 (319, 19), (320, 18)])
def test_largest_planes(gpu, oracle_lib, P, R):
    wl = slice_workload(P, R)
    flags = dict(wl.flags, run_convection=1, run_radial=0, run_local=0)
    st = O.OracleStepper(dict(W.oracle_inputs(wl), flags=flags), oracle_lib)
    st.step(wl.dt, wl.sub_dt, True)
    for arith in ("exact", "stream"):
        c = load_ctx(wl)
        c.set_convection_arith(arith)
        c.convection(wl.dt)
        c.sync()
        got = c.download()
        c.close()
        if arith == "exact":
            assert np.array_equal(got, st.psd)
        else:
            assert np.abs(got - st.psd).max() <= TOL * np.abs(st.psd).max()


@pytest.mark.parametrize("arith,P,R", [("exact", 99, 134), ("exact", 228, 51), ("fma", 64, 128),
                                       ("fma", 53, 291)])
def test_line_kernels_limit(gpu, arith, P, R):
    wl = slice_workload(P, R)
    c = load_ctx(wl)
    c.set_convection_arith(arith)
    with pytest.raises(VerbError) as e:
        c.convection(wl.dt)
    c.close()
    assert "VERB_ERR_SIZE" in str(e.value)
