"""The surrogate's training step: the gradient kernel at the edges of its
tiles (16 rows a warp, 128 a CTA, more rows than one wave of CTAs), and the
update kernel's Adam step and packed weights."""
import numpy as np
import pytest

from oracle import mlp_ref

pytestmark = pytest.mark.gpu

POTENTIAL = "4*(r**-12-r**-6) + 0.5*exp(-(r-1.5)**2/0.02) + 0.1*cos(4*r)*exp(-r)"


def _surrogate(n_samples=4096, seed=5):
    from dompap_gb300.mlp import PairSurrogate

    sur = PairSurrogate(POTENTIAL, 3.0, n_samples=n_samples, seed=seed)
    sur.set_params(np.random.default_rng(2).normal(0, 0.3, sur.nparam).astype(np.float32))
    return sur


@pytest.mark.parametrize("n", [1, 7, 8, 9, 15, 16, 17, 127, 128, 129, 1000, 152 * 4 * 128 + 5])
@pytest.mark.parametrize("accurate", [True, False])
def test_gradient_at_tile_edges(n, accurate):
    sur = _surrogate()
    rng = np.random.default_rng(n)
    s = (rng.uniform(0.8, 3.0, n) ** 2).astype(np.float32)
    t = rng.normal(0, 1, (n, 2)).astype(np.float32)
    x = (s.astype(np.float64) - float(sur.norm[0])) * float(sur.norm[1])
    loss, g = sur.gradients(s, t, wf=0.7, accurate=accurate)
    loss_ref, g_ref = mlp_ref.loss_and_grad(sur.params(), x, t.astype(np.float64), wf=0.7)
    # bf16 operands of the backward products (2^-9 each) and, not accurate, the
    # hardware tanh (2^-11): a few of these in the L2 norm
    assert abs(loss - loss_ref) <= 5e-3 * loss_ref
    for sl in (slice(0, 64), slice(64, 128), slice(128, 4224), slice(4224, 4288), slice(4288, 4416), slice(4416, 4418)):
        assert np.linalg.norm(g[sl] - g_ref[sl]) <= 3e-2 * np.linalg.norm(g_ref[sl])


def test_step_is_adam_on_the_drawn_samples_and_packs_its_weights():
    """Batch = all samples drawn with replacement: the step moves every weight
    by the learning rate against its gradient's sign on the first step
    (Adam's bias correction), the loss it reports is the batch's, and the
    packed network is the one a fresh set_params of the new weights gives."""
    sur = _surrogate()
    before = sur.params()
    loss = sur.train(1, batch=129, lr0=1e-3, lr1=1e-3)
    after = sur.params()
    moved = np.abs(after - before)
    # |m / (sqrt(v) + 1e-8)| = |g| / (|g| + 1e-8): the learning rate wherever the
    # gradient is not tiny, never more (plus the weights' own rounding)
    assert np.max(moved) <= 1e-3 * (1 + 1e-5) + 3e-7
    assert np.median(moved) >= 0.99e-3
    assert np.isfinite(loss[0]) and loss[0] > 0
    for steps in (1, 5):
        sur.train(steps, batch=500)
        fresh = _surrogate()
        fresh.set_params(sur.params())
        s = np.linspace(0.7, 9.0, 777).astype(np.float32)
        assert np.array_equal(sur.network(s), fresh.network(s))
        t = np.zeros((777, 2), dtype=np.float32)
        g, h = sur.gradients(s, t)[1], fresh.gradients(s, t)[1]  # forward and transposed fragments
        assert np.array_equal(g, h)


def test_training_is_reproducible_and_splits():
    """Bit for bit: two surrogates, and one run against the same steps in parts
    (a constant learning rate, since each call has its own schedule)."""
    a, b = _surrogate(), _surrogate()
    la = a.train(12, batch=1000, lr0=1e-3, lr1=1e-3)
    lb = np.concatenate([b.train(5, batch=1000, lr0=1e-3, lr1=1e-3), b.train(7, batch=1000, lr0=1e-3, lr1=1e-3)])
    assert np.array_equal(a.params(), b.params()) and np.array_equal(la, lb)


@pytest.mark.parametrize("scale", [1.0, 30.0, 1000.0])
def test_gradient_sums_of_small_and_large_terms(scale):
    """Terms on both sides of 2^31 fixed-point units (1/32 of a gradient, 1/2 of
    a loss): the 32-bit and the shifted conversion, both signs."""
    sur = _surrogate()
    rng = np.random.default_rng(11)
    n = 129
    s = (rng.uniform(0.8, 3.0, n) ** 2).astype(np.float32)
    t = (scale * rng.normal(0, 1, (n, 2))).astype(np.float32)
    x = (s.astype(np.float64) - float(sur.norm[0])) * float(sur.norm[1])
    loss, g = sur.gradients(s, t, wf=0.7, accurate=True)
    loss_ref, g_ref = mlp_ref.loss_and_grad(sur.params(), x, t.astype(np.float64), wf=0.7)
    # as at the tile edges: bf16 operands of the backward products, 2^-9 each
    assert abs(loss - loss_ref) <= 5e-3 * loss_ref
    for sl in (slice(0, 64), slice(64, 128), slice(128, 4224), slice(4224, 4288), slice(4288, 4416), slice(4416, 4418)):
        assert np.linalg.norm(g[sl] - g_ref[sl]) <= 3e-2 * np.linalg.norm(g_ref[sl])
