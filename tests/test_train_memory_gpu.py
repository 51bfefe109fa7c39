"""The gradient call on the tensor-core training kernels holds what those kernels
use: a row's inputs and targets, its share of the tiles between the kernels (six of
64 KiB a 128-row tile) and of the edge partials (four rows of 4,104 floats a tile),
and, whatever the rows, two layers' derivatives a CTA and the weight gradients'
partials of at most 64 shares.  None of the layer-by-layer path's 10 KB a row.

The bound is that sum and a tenth for the allocator's granularity.  A forward call
of the same size after it (which does use the layer-by-layer buffers) and a smaller
gradient call still agree with calls of an object of their own.
"""
from contextlib import closing

import numpy as np
import pytest

from spacetime_gb300.surrogate import Surrogate

pytestmark = pytest.mark.gpu


def test_gradient_call_holds_what_it_uses(built_lib):
    torch = pytest.importorskip("torch")
    n = 262144
    rng = np.random.default_rng(0)
    X = rng.uniform(-1, 1, (n, 6)).astype(np.float32)
    T = rng.uniform(-1, 1, (n, 8)).astype(np.float32)
    with closing(Surrogate(0, seed=5)) as s, closing(Surrogate(0, seed=5)) as other:
        free = torch.cuda.mem_get_info()[0]
        s.loss_grad(X, T)
        held = free - torch.cuda.mem_get_info()[0]
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        want = n * (14 * 4 + 6 * 65536 // 128 + 4 * 4104 * 4 // 128) + sms * 2 * 256 * 128 * 4 + 64 * 3 * 65536 * 4
        assert held <= 1.1 * want, (held, want)
        np.testing.assert_array_equal(s.forward(X[:1000]), other.forward(X[:1000]))
        a, b = s.loss_grad(X[:300], T[:300]), other.loss_grad(X[:300], T[:300])
        np.testing.assert_array_equal(a[1], b[1])
        np.testing.assert_array_equal(s.forward(X), other.forward(X))
