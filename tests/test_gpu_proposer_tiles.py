"""The proposer's network kernel at the edges of its tiles: one to a few
examples, one more or less than a block's, and a ragged last block."""
import numpy as np
import pytest

import poa_b200
from tests import proposer_net as net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 4, 5, 7, 147, 149, 593])
def test_predict_and_gradient_at_remainders(n):
    w, X, Y = net.random_problem(100 + n, n)
    X, Y = X.astype(np.float32), Y.astype(np.float32)
    prop = poa_b200.Proposer()
    prop.set_weights(w.astype(np.float32))
    w64 = prop.get_weights().astype(np.float64)
    got, want = prop.predict(X), net.predict(w64, X, use_bf16=True)
    # the same BF16 rounding points, float32 sums in another order
    assert np.all(np.abs(got - want) <= 2e-2 * (np.std(want, axis=0) + 1e-3)[None, :])
    loss, g = prop.gradient(X, Y)
    want_loss, wg = net.loss_and_gradient(w64, X, Y, use_bf16=True)
    assert abs(loss - want_loss) <= 1e-3 * abs(want_loss) + 1e-6
    o = 0
    for name, shape in net.SHAPES:
        k = int(np.prod(shape))
        a, b = g[o:o + k].astype(np.float64), wg[o:o + k]
        o += k
        assert np.linalg.norm(a - b) <= 2e-2 * (np.linalg.norm(b) + 1e-12), name


def test_examples_do_not_depend_on_their_place():
    """A batch's predictions are each example's own, whatever block and lane it fell on."""
    w, X, _ = net.random_problem(5, 300)
    X = X.astype(np.float32)
    prop = poa_b200.Proposer()
    prop.set_weights(w.astype(np.float32))
    whole = prop.predict(X)
    for a, b in ((0, 1), (1, 4), (17, 166), (150, 300)):
        np.testing.assert_array_equal(prop.predict(X[a:b]), whole[a:b])
