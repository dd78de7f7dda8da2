"""Per-slice operators keep idle device blocks between calls: calls of growing
and shrinking sizes in turn, from several host threads at once, and after one
that fails give the results of the same calls one by one (which
tests/test_gpu_ops.py holds to the reference)."""
import threading

import numpy as np
import pytest

from verb4d_b200 import VerbError, ops
from verb4d_b200 import workload as W

pytestmark = pytest.mark.gpu


def convection_call(P, R, seed):
    wl = W.make_workload(W.GridSpec(P, R, 1, 1), seed=seed, sources=True)
    q = lambda n: np.ascontiguousarray(wl.fields[n][:, :, 0, 0])  # noqa: E731
    f, t = wl.fields, wl.bc_types
    args = (q("psd"), q("Pg"), q("Rg"), P, R, f["Pl"][:, 0, 0].copy(), f["Pu"][:, 0, 0].copy(),
            f["Rl"][:, 0, 0].copy(), f["Ru"][:, 0, 0].copy(), t["Pl"], t["Pu"], t["Rl"], t["Ru"],
            q("VP"), q("VR"), q("S"), q("loss_conv"), q("G_conv"), wl.dt)
    return lambda: ops.Convection_2D(*args)


def diffusion_call(V, K, seed):
    wl = W.make_workload(W.GridSpec(1, 1, V, K), seed=seed, sources=True)
    f, t = wl.fields, wl.bc_types
    q = lambda n: np.ascontiguousarray(f[n][0, 0])  # noqa: E731
    args = (q("psd"), q("Vg"), q("Kg"), V, K, f["Vl"][0, 0], f["Vu"][0, 0], f["Kl"][0, 0],
            f["Ku"][0, 0], t["Vl"], t["Vu"], t["Kl"], t["Ku"], q("DVV"), q("DKK"), q("DVK"),
            q("DVK"), q("G_local"), q("S"), q("loss_local"), wl.dt, wl.sub_dt)
    return lambda: ops.Diffusion_2D(*args)


def tridag_call(n, seed):
    rng = np.random.default_rng(seed)
    a, b, c, r = rng.uniform(0.1, 1, (4, n))
    return lambda: ops.tridag(a, b + 3, c, r)


def test_sizes_in_turn_and_threads(gpu):
    calls = [convection_call(12, 13, 1), diffusion_call(31, 31, 2), tridag_call(5, 3),
             diffusion_call(9, 9, 4), convection_call(48, 101, 5), tridag_call(20000, 6),
             diffusion_call(61, 40, 7), convection_call(24, 25, 8)]
    ref = [f() for f in calls]
    for _ in range(2):
        for f, x in reversed(list(zip(calls, ref))):
            assert np.array_equal(f(), x)
    bad = []

    def work(i):
        for k in range(12):
            j = (i * 3 + k) % len(calls)
            if not np.array_equal(calls[j](), ref[j]):
                bad.append((i, j))

    th = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad
    with pytest.raises(VerbError):  # Courant failure: a zero grid spacing
        ops.Convection_1D(np.ones(12), np.zeros(12), 12, 0.0, 0.0, 1, 1, np.ones(12), 1.0)
    for f, x in zip(calls, ref):
        assert np.array_equal(f(), x)
