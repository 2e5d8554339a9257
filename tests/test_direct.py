"""kfmm_direct_evaluation at the edges of its tiles and splits (GPU).

The pair term's reciprocal square root is checked over the whole exponent range
against extended precision, and the sums at target and source counts around
the kernel's tile of 32 targets and its source splits (4, 16 and 128 shares of
at least four 32-source chunks).
"""
import numpy as np
import pytest

EPS = 2.0 ** -52


def _direct(K, t, s, start=0.0):
    import torch
    T = [torch.tensor(np.ascontiguousarray(v), device="cuda:0") for v in t]
    S = [torch.tensor(np.ascontiguousarray(v), device="cuda:0") for v in s]
    pot = torch.full((len(t[0]),), start, dtype=torch.float64, device="cuda:0")
    K.check(K.lib().kfmm_direct_evaluation(len(t[0]), *[x.data_ptr() for x in T], pot.data_ptr(),
                                           len(s[0]), *[x.data_ptr() for x in S], None), "direct")
    torch.cuda.synchronize()
    return pot.cpu().numpy()


@pytest.mark.gpu
def test_pair_term_accuracy(K, cuda_ok):
    """One source at the origin, targets on the x axis from 1e-140 to 1e140:
    1/(4 pi r) within 3 eps.  Roundings, in units of eps/2: r^2 (half of it
    reaches the root) 0.5, the root 2, the constant 1, the last product 1."""
    rng = np.random.default_rng(1)
    x = 10.0 ** rng.uniform(-140, 140, 200000) * rng.choice([-1.0, 1.0], 200000)
    z = np.zeros_like(x)
    got = _direct(K, (x, z, z), tuple(np.array([v]) for v in (0.0, 0.0, 0.0, 1.0)))
    pi = np.longdouble("3.14159265358979323846264338327950288")
    ref = 1.0 / (4.0 * pi * np.abs(x.astype(np.longdouble)))
    err = np.abs(got.astype(np.longdouble) - ref) / ref
    print(f"max relative error {float(err.max()) / EPS:.2f} eps")
    assert float(err.max()) <= 3 * EPS


@pytest.mark.gpu
def test_tiny_distances(K, cuda_ok):
    """The same bound down to the smallest r whose square is a normal number
    (1.5e-154), in the direct sum and between the points of one leaf."""
    rng = np.random.default_rng(2)
    r = 10.0 ** rng.uniform(-153.7, -140, 20000)
    x = r * rng.choice([-1.0, 1.0], r.size)
    z, one = np.zeros_like(x), tuple(np.array([v]) for v in (0.0, 0.0, 0.0, 1.0))
    ref = 1.0 / (4 * np.pi * r.astype(np.longdouble))
    got = _direct(K, (x, z, z), one)
    assert float(np.max(np.abs(got - ref) / ref)) <= 3 * EPS
    pts = dict(zip(("sx", "sy", "sz", "den"), one), tx=x, ty=z, tz=z)
    tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], 64)
    assert tree.desc.num_nodes == 1
    got = K.Plan(tree, 4, K.PLAIN_FP64).evaluate(pts)
    assert float(np.max(np.abs(got - ref) / ref)) <= 3 * EPS


@pytest.mark.gpu
def test_skipped_pairs(K, cuda_ok):
    """Coincident points, sources at infinity and at NaN add nothing."""
    t = np.array([[0.25, 0.5], [0.5, 0.5], [-0.5, 0.125]])
    s = np.array([[0.25, np.inf, np.nan, 0.75], [0.5, 0.0, 0.0, 0.5], [-0.5, 0.0, 0.0, -0.5],
                  [3.0, 2.0, 5.0, 1.0]])
    got = _direct(K, t, s, 1.0)
    ref = np.ones(2)
    for i in range(2):
        for j in (0, 3):
            r = np.sqrt(((t[:, i] - s[:3, j]) ** 2).sum())
            if r > 0:
                ref[i] += s[3, j] / (4 * np.pi * r)
    assert np.allclose(got, ref, rtol=1e-14, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("ns", [1, 31, 33, 511, 512, 2048, 2049, 16383, 16384, 20001])
@pytest.mark.parametrize("nt", [1, 32, 33, 700, 9473])
def test_split_edges(K, cuda_ok, nt, ns):
    """Positive densities: any order of n sums of positive terms is within
    n eps of another; sqrt(n) + 8 bounds what is seen with room."""
    rng = np.random.default_rng(nt * 7 + ns)
    t, s = rng.uniform(-1, 1, (3, nt)), rng.uniform(-1, 1, (4, ns))
    s[3] = np.abs(s[3])
    m = min(nt, ns, 5)
    s[:3, :m] = t[:, :m]
    got = _direct(K, t, s, 0.5)
    pick = np.unique(np.concatenate([np.arange(min(nt, 40)), np.arange(max(0, nt - 40), nt)]))
    r = np.sqrt(((t[:, pick, None] - s[:3, None, :]) ** 2).sum(0))
    ref = 0.5 + (np.where(r > 0, 1.0 / np.where(r > 0, r, 1.0), 0.0) @ s[3]) / (4 * np.pi)
    assert np.max(np.abs(got[pick] - ref) / ref) <= (np.sqrt(ns) + 8) * EPS
    assert np.all(np.isfinite(got))
