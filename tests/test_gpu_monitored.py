"""Monitored steps: the slots a handle keeps for them and the blocks of steps
that share a memset and a copy (lbm_step_monitored copies its results to the
host every 4096 steps)."""
import numpy as np
import pytest

from cudalbm_b200 import _lib
from cudalbm_b200.solver import Cavity

pytestmark = pytest.mark.gpu

BLOCK = 4096


def same_sums(a, b):
    # the sums are atomic FP64 additions: equal up to their order
    np.testing.assert_allclose(a["mass"], b["mass"], rtol=1e-12)
    np.testing.assert_allclose(a["rho_u2"], b["rho_u2"], rtol=1e-12)
    assert np.array_equal(a["nonfinite"], b["nonfinite"])


def test_monitored_calls_allocate_nothing():
    """The first monitored call of a handle, and a longer later one, find
    their slots: device memory is what it was after creation."""
    with Cavity(19, 16, 16, 16, 100.0, 0.05) as c:
        c.init_regions()
        before = c.info()["device_bytes"]
        for n in (1, 100, BLOCK + 1):
            c.step_monitored(n)
            c.synchronize()
            assert c.info()["device_bytes"] == before, n


@pytest.mark.parametrize("n", [BLOCK - 1, BLOCK, BLOCK + 1, 2 * BLOCK + 3])
def test_results_across_blocks_of_steps(n):
    """Calls that end before, on and past the end of a block: the sums of
    every step as from calls of other lengths, the state as from plain steps."""
    with Cavity(19, 16, 8, 8, 100.0, 0.05) as a, Cavity(19, 16, 8, 8, 100.0, 0.05) as b, \
            Cavity(19, 16, 8, 8, 100.0, 0.05) as plain:
        for c in (a, b, plain):
            c.init_regions()
        whole = a.step_monitored(n)
        parts = [b.step_monitored(k) for k in (1000, 77, n - 1077)]
        plain.step(n)
        for c in (a, b, plain):
            c.synchronize()
        same_sums(whole, np.concatenate(parts))
        assert np.all(whole["mass"] > 0.0)
        ref = plain.read()
        for c in (a, b):
            assert np.array_equal(c.read().view(np.uint32), ref.view(np.uint32))


def test_streamed_job_longer_than_a_block():
    """A monitored streamed job of more steps than the handle has slots, and a
    monitored call after it."""
    n = BLOCK + 5
    with Cavity(19, 16, 8, 8, 100.0, 0.05) as a, Cavity(19, 16, 8, 8, 100.0, 0.05) as b:
        for c in (a, b):
            c.init_regions()
        state = a.read()
        out, mon = np.empty_like(state), np.zeros(n, _lib.MONITOR_DTYPE)
        a.run_streamed(state, n, {"moments": out}, monitor=mon)
        ref = b.step_monitored(n)
        b.synchronize()
        same_sums(mon, ref)
        assert np.array_equal(out.view(np.uint32), b.read().view(np.uint32))
        x, y = a.step_monitored(3), b.step_monitored(3)
        a.synchronize()
        b.synchronize()
        same_sums(x, y)
