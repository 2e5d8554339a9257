"""The cost-model network's kernels at the edges of their 64 x 64 tiles, 16-deep
slices and batch ranges (GPU), against the FP64 oracle."""
import mlp_oracle as MO
import numpy as np
import pytest

EPS = 2.0 ** -23


@pytest.mark.gpu
@pytest.mark.parametrize("F,H,O,B", [(1, 1, 1, 1), (16, 64, 5, 63), (17, 63, 64, 65),
                                     (73, 64, 5, 4097), (65, 129, 65, 200), (64, 15, 1, 10000)])
def test_gradients_at_tile_edges(K, cuda_ok, F, H, O, B):
    """Every output within 8 sqrt(n) eps of the scale of its terms' sum, n the
    longest chain of sums on its way (F, H, H forward, O, H backward, B over the
    batch; roundings of random sign); a hidden unit within rounding of zero may
    switch, which the batch's largest single term (1 / B) covers."""
    rng = np.random.default_rng(F + H + O + B)
    n = F * H + H + H * H + H + H * O + O
    p = (0.3 * rng.standard_normal(n)).astype(np.float32)
    X = rng.standard_normal((B, F)).astype(np.float32)
    T = rng.standard_normal((B, O)).astype(np.float32)
    net = K.MLP(F, H, O, params=p)
    Y = net.forward(X)
    Yo, _ = MO.forward(p.astype(np.float64), X, F, H, O)
    assert np.max(np.abs(Y - Yo)) <= 8 * np.sqrt(F + 2 * H) * EPS * np.max(np.abs(Yo))
    g, loss = net.gradients(X, T)
    lo, go = MO.loss_and_gradients(p.astype(np.float64), X, T, F, H, O)
    chain = 8 * np.sqrt(F + 3 * H + O + B) * EPS
    assert abs(loss - lo) <= chain * lo
    assert np.max(np.abs(g - go)) <= chain * np.max(np.abs(go))


@pytest.mark.gpu
def test_training_steps_follow_the_oracle(K, cuda_ok):
    """Five Adam steps from the same parameters: losses to FP32 rounding,
    parameters to a small share of one step (lr), and losses=NULL accepted."""
    import ctypes
    F, H, O, B, lr = 9, 64, 3, 1000, 2e-3
    rng = np.random.default_rng(3)
    n = F * H + H + H * H + H + H * O + O
    p0 = (0.2 * rng.standard_normal(n)).astype(np.float32)
    X = rng.standard_normal((B, F)).astype(np.float32)
    T = np.tanh(X[:, :O]).astype(np.float32)
    net = K.MLP(F, H, O, params=p0.copy())
    losses = net.train(X, T, 5, lr)
    p, m, v, want = p0.astype(np.float64), np.zeros(n), np.zeros(n), []
    for s in range(1, 6):
        loss, g = MO.loss_and_gradients(p, X, T, F, H, O)
        want.append(loss)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - lr * (m / (1 - 0.9 ** s)) / (np.sqrt(v / (1 - 0.999 ** s)) + 1e-8)
    assert np.allclose(losses, want, rtol=1e-5)
    assert np.linalg.norm(net.params - p) <= 0.01 * lr * np.sqrt(n)
    again = p0.copy()
    f32 = ctypes.POINTER(ctypes.c_float)
    K.check(K.lib().kfmm_mlp_train(F, H, O, again.ctypes.data_as(f32), B, X.ctypes.data_as(f32),
                                   T.ctypes.data_as(f32), 5, lr, None), "train")
    assert np.array_equal(again, net.params)
