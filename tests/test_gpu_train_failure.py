"""A bounded wait of the training kernel that runs out (the test hook shortens each CTA's
first one): the call returns, the failure is counted and reported, no parameter changes,
and the next batch gives the normal result.  Batches of one CTA, of one tile a CTA, and
of several tiles a CTA.

The failed launches' reads and writes stay in bounds and all their products end before
the CTA does: only the values of the tile that gave up are wrong, and they are left out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [100, 16384, 45000])
def test_training_wait_that_runs_out(gi, cuda, n):
    r = np.random.default_rng(n)
    x = cuda.from_numpy(r.uniform(0.0, 1.0, (n, 32)).astype(np.float32)).cuda().bfloat16()
    t = cuda.from_numpy(r.uniform(0.0, 1.0, (n, 4)).astype(np.float32)).cuda()
    net, fresh = gi.Mlp(seed=5), gi.Mlp(seed=5)
    loss, grads = net.gradients(x, t)
    before = net.get_params()
    errors = gi.tensor_core_errors()
    try:
        gi.debug_tensor_core_wait_limit(1)
        for call in (lambda: net.gradients(x, t), lambda: net.train_step(x, t)):
            with pytest.raises(gi.GiError) as e:
                call()
            assert e.value.status == gi.GI_ERR_TIMEOUT
            assert gi.tensor_core_errors() > errors
            errors = gi.tensor_core_errors()
        fresh.train_step(x, t, want_loss=False)  # reports nothing, changes nothing
        cuda.cuda.synchronize()
        assert gi.tensor_core_errors() > errors
        errors = gi.tensor_core_errors()
    finally:
        gi.debug_tensor_core_wait_limit(0)
    np.testing.assert_array_equal(net.get_params(), before)
    np.testing.assert_array_equal(fresh.get_params(), before)
    # FP32 sums of up to 152 CTAs in any order: 152 * 2^-24 of a sum of magnitudes, 1e-4 with
    # cancellation of a factor of ten.
    loss2, grads2 = net.gradients(x, t)
    assert abs(loss2 - loss) <= 1e-4 * abs(loss)
    assert np.abs(grads2 - grads).max() <= 1e-4 * np.abs(grads).max()
    # The step after a failed one is a first step: Adam moves a parameter by lr times the
    # sign of its gradient (to eps / |gradient|), where that is not lost in the sums' order.
    net.train_step(x, t, lr=1e-3)
    moved = net.get_params() - before
    clear = np.abs(grads) > 1e-3 * np.abs(grads).max()
    assert clear.sum() > 100
    np.testing.assert_allclose(moved[clear], -1e-3 * np.sign(grads[clear]), rtol=2e-2)
    assert gi.tensor_core_errors() == errors
