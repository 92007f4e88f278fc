"""Gradients at batch sizes around the tile of 128 rows, the groups of the
column sums and the blocks of the embedding gradient, against the float64
oracle (the same tolerances as at 256 examples: loss 1e-3, each tensor 2e-2
relative L2; a tensor no example reaches is zero on both sides)."""
import numpy as np
import pytest

import mlp_ref
from m6502.mlp import MLP
from test_gpu_mlp import _examples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 127, 129, 513, 1300])
def test_gradients_at_ragged_sizes(engine, n):
    mlp = MLP(engine, seed=n)
    ex = _examples(n, n)
    loss, g = mlp.gradients(ex)
    ref_loss, ref = mlp_ref.loss_and_grads(ex, mlp.params())
    assert abs(loss - ref_loss) <= 1e-3 * abs(ref_loss)
    o = 0
    for i, (r, c) in enumerate(mlp_ref.SHAPES):
        got = g[o:o + r * c].astype(np.float64).reshape(ref[i].shape)
        o += r * c
        assert np.linalg.norm(got - ref[i]) <= 2e-2 * np.linalg.norm(ref[i]), i
    mlp.close()
