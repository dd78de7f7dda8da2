"""Per-slice operators on sizes whose block of device memory (sized for every
phase of a context) would be larger than the device: the answer is the one the
call has by itself, and the next call is not disturbed."""
import numpy as np
import pytest

from verb4d_b200 import VerbError, ops
from test_gpu_ops_threads import diffusion_call

pytestmark = pytest.mark.gpu


def test_wide_band_refused_as_such(gpu):
    small = diffusion_call(9, 9, 4)
    ref = small()
    V, K = 20000, 24  # factors of 230 GB, if the band were solved at all
    z, e, x = np.zeros((V, K)), np.zeros(max(V, K)), np.ones((V, K))
    with pytest.raises(VerbError) as err:
        ops.Diffusion_2D(z, x, x, V, K, e[:K], e[:K], e[:V], e[:V], 1, 1, 1, 1, x, x, z, z, x, z, z,
                         1.0, 1.0)
    assert err.value.status == 2
    assert np.array_equal(small(), ref)

