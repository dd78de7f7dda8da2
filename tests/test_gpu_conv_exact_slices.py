"""The exact convection over its rule on the number of slices: both sides of
the small slices' limit of two an SM, one, two and three slices resident on an
SM, and the counts at which slices of more points go back to the line-job
kernel.  Bit for bit against the oracle (no convection losses: exp() may differ
in the last bit from the host's)."""
import numpy as np
import pytest

from verb4d_b200 import workload as W

from test_gpu_conv_staged_exact import check
from test_gpu_conv_stream import BCS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,R,V,K", [(12, 13, 37, 8), (12, 13, 27, 11), (12, 13, 50, 30),
                                     (13, 12, 60, 61), (24, 25, 37, 32), (24, 25, 35, 34),
                                     (20, 21, 64, 38), (24, 51, 37, 32), (24, 51, 35, 34),
                                     (36, 50, 48, 37), (36, 50, 61, 30)])
def test_slice_counts(gpu, oracle_lib, P, R, V, K):
    wl = W.make_workload(W.GridSpec(P, R, V, K), seed=V, sources=True)
    wl.fields["VP"] = wl.fields["VP"] * 0.02
    wl.bc_types.update(Pl=BCS["periodic"], Pu=BCS["periodic"])
    check(wl, oracle_lib)
