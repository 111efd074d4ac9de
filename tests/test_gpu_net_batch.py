"""Gradients of the warm-start network at extents around its kernels' tiles, and
their accumulation over a training batch: a batch that holds one sample
twice has the sums 2 g and 2 loss, exact in binary arithmetic, so its mean
loss and the updated parameters equal those of the sample alone bit for bit;
and the loss and gradient do not depend on what ran before."""
import numpy as np
import pytest

import ofblend_gb300 as F
from oracle import warmstart_net as W

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


@pytest.mark.parametrize("R", [20, 28])
def test_gradient_matches_oracle_beyond_one_tile(gpu, R):
    """20^4 has levels 20, 10 and 5, no multiple of the halo tiles' 8 x 16
    voxels; at 28^4 the 96-column input gradient no longer fits two halo
    stages and takes the im2col kernel."""
    m = F.Model(R, seed=8)
    p = W.bf16_round(m.get_params())
    m.set_params(p)
    r = np.random.default_rng(R)
    d = (R,) * 4
    i0 = (r.standard_normal(d) * 0.004).astype(np.float32)
    i1 = (r.standard_normal(d) * 0.004).astype(np.float32)
    tgt = (r.standard_normal(d + (4,)) * 0.5).astype(np.float32)
    loss, g = m.loss_grad(F.Grid4Real(dims=d).from_numpy(i0), F.Grid4Real(dims=d).from_numpy(i1),
                          F.Grid4Vec4(dims=d).from_numpy(tgt))
    wloss, wg = W.loss_and_grad(p, i0, i1, tgt)
    assert abs(loss - wloss) <= 1e-4 * abs(wloss)
    # as test_gpu_warmstart.py: 1e-3 of a block, but the first layer's weights
    # and bias 1e-2: one activation on the other side of zero moves them by
    # about the inverse root of the voxels (160000: 2.5e-3) of their norm
    off, gnorm = 0, np.linalg.norm(wg)
    for l, (cin, cout, ks, *_) in enumerate(W.LAYERS):
        for n in ((81 if ks == 3 else 1) * cin * cout, cout):
            a, b = g[off:off + n].astype(np.float64), wg[off:off + n]
            tol = 1e-2 if l == 0 else 2e-3
            assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b) + 1e-7 * gnorm, (l, n)
            off += n
