"""The solve at the sizes where its kernels' shapes change (GPU).

Near field: leaves of one target up to several rows of 32, around the team jobs'
copies (8 and 16 targets), their split rows (32, 64, 128) and remainders.  A
single leaf's potentials are the direct sum, which FP64 NumPy gives.

Far field: trees of a few hundred boxes at every NP, against the oracle:
few V-list windows (shared by several warps of the Hadamard kernels) and level
products of few columns, operators whose sizes leave remainders in every tile.
"""
import numpy as np
import pytest

SIZES = [1, 7, 8, 9, 16, 17, 31, 32, 33, 47, 48, 49, 64, 65, 81, 127, 128, 129, 144, 145, 200, 421]


def _direct(pts):
    t = np.stack([pts[k] for k in ("tx", "ty", "tz")])
    s = np.stack([pts[k] for k in ("sx", "sy", "sz")])
    r = np.sqrt(((t[:, :, None] - s[:, None, :]) ** 2).sum(0))
    inv = np.where(r > 0, 1.0 / np.where(r > 0, r, 1.0), 0.0)
    return inv @ pts["den"] / (4 * np.pi)


@pytest.mark.gpu
@pytest.mark.parametrize("coincide", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_single_leaf(K, cuda_ok, n, coincide):
    """Positive densities.  Plain: n eps at most, sqrt(n) + 8 with room.  Mixed:
    coordinates and pair terms in FP32 relative to a box of radius 1, so a pair
    at distance r is off by about 2^-24 / r; the closest pair bounds it."""
    if n == 1 and coincide:
        pytest.skip("no pair")
    pts = K.generate_points(n, "uniform", coincide, 11 + n)
    tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], n)
    assert tree.desc.num_nodes == 1
    ref = _direct(pts)
    plain = K.Plan(tree, 4, K.PLAIN_FP64).evaluate(pts)
    assert np.max(np.abs(plain - ref) / ref) <= (np.sqrt(n) + 8) * 2.0 ** -52
    t = np.stack([pts[k] for k in ("tx", "ty", "tz")])
    s = np.stack([pts[k] for k in ("sx", "sy", "sz")])
    r = np.sqrt(((t[:, :, None] - s[:, None, :]) ** 2).sum(0))
    near = r[r > 0].min()
    mixed = K.Plan(tree, 4, K.MIXED).evaluate(pts)
    assert np.max(np.abs(mixed - ref) / ref) <= 8 * 2.0 ** -24 * (1 + 1 / near)


@pytest.mark.gpu
@pytest.mark.parametrize("dist,n,ppb", [("uniform", 1500, 20), ("ellipsoidSurface", 1200, 12)])
@pytest.mark.parametrize("np_", [3, 4, 5, 6, 7, 8])
def test_few_boxes_vs_oracle(K, oracle_mod, cuda_ok, np_, dist, n, ppb):
    """Potentials of both forms against the oracle; plain within 1e-12 or twice
    the oracle's own change when its sums are reversed."""
    pts = K.generate_points(n, dist, 0, 26)
    tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], ppb)
    tarrs = {k: tree.array(k) for k in oracle_mod.TREE_FIELDS}
    ops = K.operators(np_)
    ref = oracle_mod.evaluate(tarrs, np_, ops, pts)
    back = oracle_mod.evaluate_reordered(tarrs, np_, ops, pts)
    scale = np.abs(ref).max()
    floor = np.max(np.abs(back - ref)) / scale
    plain = K.Plan(tree, np_, K.PLAIN_FP64).evaluate(pts)
    assert np.max(np.abs(plain - ref)) / scale <= max(1e-12, 2 * floor)
    mixed = K.Plan(tree, np_, K.MIXED).evaluate(pts)
    err = np.linalg.norm(mixed - ref) / np.linalg.norm(ref)
    # FP32 pair terms and spectra: 2e-7 on uniform clouds; crowded poles and
    # cancelling densities leave 3e-5 on the ellipsoid surface
    assert err <= (1e-6 if dist == "uniform" else 1e-4)
