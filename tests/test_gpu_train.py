"""The training pass of the learned layer's network at the edges of its
decomposition: 128 samples per pass, any number of passes.
"""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from oracle.oracle import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def samples(n, seed):
    s = mo.random_samples(n, seed)
    s[1::4, :32] = 0.0  # silent samples contribute nothing
    rng = np.random.default_rng(seed + 1)
    r = np.sqrt(np.mean(s[:, :32].astype(np.float64) ** 2, axis=1))
    t = (rng.normal(0, 1, (n, 2)) * (r[:, None] + 0.1)).astype(np.float32)
    return s, t


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 152 * 32 + 1, 2 * 152 * 32 + 77])
def test_gradient_sizes(dc, n):
    """Against the oracle: the hardware's tanh (2^-11) moves some BF16
    roundings (2^-9) of a sample's 64 activations, a per cent at worst for a
    few samples, averaging out over many.  Against the sum of two parts: the
    same activations, FP32 sums in another order."""
    p = mo.init_params(3)
    s, t = samples(n, 40 + n)
    xs, ts = dev(s), dev(t)
    with dc.MLP(device=0, params=p) as m:
        g, (le, lw) = m.gradient(xs.data_ptr(), ts.data_ptr(), n)
        k = n // 3
        if k:
            ga, la = m.gradient(xs.data_ptr(), ts.data_ptr(), k)
            gb, lb = m.gradient(xs.data_ptr() + k * 33 * 4, ts.data_ptr() + k * 2 * 4, n - k)
            assert rel_l2(ga.astype(np.float64) + gb, g) <= 1e-5
            assert abs(la[1] + lb[1] - lw) <= 1e-9 * lw
    gw, le_w, lw_w = mo.gradient(p, s, t)
    assert rel_l2(g, gw) <= (1e-2 if n < 100 else 2e-3)
    assert abs(lw - lw_w) <= 1e-5 * lw_w and abs(le - le_w) <= 1e-2 * le_w


@pytest.mark.parametrize("batch", [1, 33, 6000])
def test_first_adam_step(dc, batch):
    """One sample, so every drawn batch has its mean gradient g: the first
    Adam step moves each parameter by lr * g / (|g| + eps)."""
    p, lr = mo.init_params(5), 2e-3
    s, t = (a[6:7] for a in samples(7, 9))  # (the first rows are silent)
    assert np.any(s[:, :32])
    xs, ts = dev(s), dev(t)
    with dc.MLP(device=0, params=p) as m:
        g, (le, lw) = m.gradient(xs.data_ptr(), ts.data_ptr(), 1)
        hist = m.train(xs.data_ptr(), ts.data_ptr(), 1, 1, batch, lr, seed=4)
        new = m.params()
        again = m.train(xs.data_ptr(), ts.data_ptr(), 1, 40, batch, lr, seed=5)
    g = g / lw
    want = p - lr * g / (np.abs(g) + 1e-8)
    big = np.abs(g) > 1e-4  # below, FP32 sums decide the ratio
    assert big.sum() > 500
    assert np.max(np.abs(new - want)[big]) <= 1e-3 * lr
    assert np.array_equal(new[g == 0], p[g == 0])
    assert abs(hist[0] - le / lw) <= 1e-5 * le / lw
    assert again[-1] < 0.5 * hist[0]  # and it goes on downhill


FULL_GRID = 152 * 16 * 128  # samples of a launch with one pass in every CTA


def many_samples(n, seed):
    """Samples of about the same size, so that each one shows in the sums."""
    rng = np.random.default_rng(seed)
    s = np.empty((n, 33), np.float32)
    s[:, :32] = rng.normal(0, 1, (n, 32)) * rng.uniform(0.5, 2.0, (n, 1))
    s[:, 32] = rng.integers(0, 8, n)
    s[1::4, :32] = 0.0
    return s, rng.normal(0, 1, (n, 2)).astype(np.float32)


def parts(m, xs, ts, n):
    """Gradient and sums of samples [0, n), at most one pass per CTA at a time."""
    g, le, lw = 0.0, 0.0, 0.0
    for k in range(0, n, FULL_GRID):
        gk, (e, w) = m.gradient(xs.data_ptr() + k * 33 * 4, ts.data_ptr() + k * 2 * 4,
                                min(FULL_GRID, n - k))
        g, le, lw = g + gk.astype(np.float64), le + e, lw + w
    return g, le, lw


@pytest.mark.parametrize("n", [FULL_GRID + 1, FULL_GRID + 129, 3 * FULL_GRID - 57])
def test_gradient_of_several_passes_per_cta(dc, n):
    """Against the same samples in launches of one pass: the same activations;
    each FP32 sum of 2432 CTAs' partials rounds by some sqrt(2432) 2^-24 = 3e-6
    of itself, and one sample of 3e5 weighs 1e-3 of a gradient that grows like
    sqrt(n), 3e-6 of the FP64 sums."""
    s, t = many_samples(n, n)
    xs, ts = dev(s), dev(t)
    with dc.MLP(device=0, params=mo.init_params(3)) as m:
        g, (le, lw) = m.gradient(xs.data_ptr(), ts.data_ptr(), n)
        gw, le_w, lw_w = parts(m, xs, ts, n)
    assert rel_l2(g, gw) <= 2e-5
    assert abs(lw - lw_w) <= 1e-9 * lw_w and abs(le - le_w) <= 1e-9 * le_w


def test_training_step_of_several_passes_per_cta(dc):
    """A batch past one pass per CTA: its mean loss and the direction of its
    first Adam step are those of the samples it draws."""
    n, batch, lr, seed = 4001, FULL_GRID + 129, 2e-3, 11
    s, t = many_samples(n, 21)
    mask = (1 << 64) - 1
    z = np.uint64((seed + 0x9E3779B97F4A7C15) & mask) ^ (
        np.arange(batch, dtype=np.uint64) * np.uint64(0x2545F4914F6CDD1D))
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    drawn = ((z ^ (z >> np.uint64(31))) % np.uint64(n)).astype(np.int64)
    p = mo.init_params(5)
    xs, ts, xd, td = dev(s), dev(t), dev(s[drawn]), dev(t[drawn])
    with dc.MLP(device=0, params=p) as m:
        g, le, lw = parts(m, xd, td, batch)
        hist = m.train(xs.data_ptr(), ts.data_ptr(), n, 1, batch, lr, seed=seed)
        new = m.params()
    assert abs(hist[0] - le / lw) <= 2.0 ** -23 * le / lw  # (stored in FP32)
    g = g / lw
    big = np.abs(g) > 1e-4
    assert big.sum() > 500
    want = p - lr * g / (np.abs(g) + 1e-8)
    assert np.max(np.abs(new - want)[big]) <= 1e-3 * lr
