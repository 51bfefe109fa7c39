"""The training kernels' mbarrier waits are bounded.  SPACETIME_GB300_TC_WAIT_OUT=1
leaves each CTA's first copy of weights unissued (a barrier that nothing completes)
with a short bound, so every CTA's first wait runs out with nothing in flight: the
kernel frees its tensor memory and returns, the call reports ST_ECUDA, and the next
call gives what it gave before.
"""
from contextlib import closing

import numpy as np
import pytest

from spacetime_gb300 import _abi
from spacetime_gb300.surrogate import Surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 200 * 128])   # one CTA; more tiles than CTAs
def test_training_wait_runs_out(built_lib, monkeypatch, n):
    rng = np.random.default_rng(n)
    X = rng.uniform(-1, 1, (n, 6)).astype(np.float32)
    T = rng.uniform(-1, 1, (n, 8)).astype(np.float32)
    with closing(Surrogate(0, seed=5)) as s:
        loss, grad = s.loss_grad(X, T)
        monkeypatch.setenv("SPACETIME_GB300_TC_WAIT_OUT", "1")
        with pytest.raises(_abi.StError) as e:
            s.loss_grad(X, T)
        assert e.value.code == _abi.ST_ECUDA
        monkeypatch.delenv("SPACETIME_GB300_TC_WAIT_OUT")
        again, g = s.loss_grad(X, T)
    np.testing.assert_array_equal(g, grad)
    np.testing.assert_allclose(again, loss, rtol=1e-5)   # the loss sums are atomic
