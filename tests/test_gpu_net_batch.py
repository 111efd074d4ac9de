"""Gradient accumulation of a training batch: a batch that holds one sample
twice has the sums 2 g and 2 loss, exact in binary arithmetic, so its mean
loss and the updated parameters equal those of the sample alone bit for bit;
and the loss and gradient do not depend on what ran before."""
import numpy as np
import pytest

import ofblend_gb300 as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [4, 12, 20])
def test_repeated_sample_is_the_sample(gpu, R):
    r = np.random.default_rng(R)
    d = (R,) * 4
    sample = (F.Grid4Real(dims=d).from_numpy((r.standard_normal(d) * 0.004).astype(np.float32)),
              F.Grid4Real(dims=d).from_numpy((r.standard_normal(d) * 0.004).astype(np.float32)),
              F.Grid4Vec4(dims=d).from_numpy((r.standard_normal(d + (4,)) * 0.5).astype(np.float32)))
    one, two = F.Model(R, seed=5), F.Model(R, seed=5)
    loss, grad = one.loss_grad(*sample)
    assert np.isfinite(grad).all() and np.abs(grad).max() > 0
    assert one.train_step([sample]) == loss
    assert two.train_step([sample, sample]) == loss
    assert np.array_equal(one.get_params(), two.get_params())
    three = F.Model(R, seed=5)
    again, g2 = three.loss_grad(*sample)
    assert again == loss and np.array_equal(g2, grad)
