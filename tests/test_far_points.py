"""Points outside every box, at infinity among them, in a plan (GPU): a source there adds
nothing to any potential (1/r = 0), in either form and in every path a source
takes (pairs, S2M, X list), and a target there disturbs no other."""
import numpy as np
import pytest

FAR = [(np.inf, 0.1, 0.2), (-np.inf, np.inf, 0.0), (1e300, -1e300, 0.5), (0.1, 0.2, -1e160)]


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["PLAIN_FP64", "MIXED"])
@pytest.mark.parametrize("dist,n,ppb,np_", [("uniform", 40, 64, 4), ("uniform", 20000, 64, 4),
                                            ("ellipseUniformAngles", 9000, 24, 3)])
def test_far_points(K, cuda_ok, form, dist, n, ppb, np_):
    pts = K.generate_points(n, dist, 0, 5)
    tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], ppb)
    plan = K.Plan(tree, np_, getattr(K, form))
    at = np.linspace(1, n - 2, len(FAR)).astype(int)
    absent = {**pts, "den": pts["den"].copy()}
    absent["den"][at] = 0.0
    want = plan.evaluate(absent)
    moved = {k: v.copy() for k, v in pts.items() if k != "check_ids"}
    for i, p in zip(at, FAR):
        moved["sx"][i], moved["sy"][i], moved["sz"][i] = p
    assert np.array_equal(plan.evaluate(moved), want)
    for i, p in zip(at, FAR):
        moved["tx"][i], moved["ty"][i], moved["tz"][i] = p
    got = plan.evaluate(moved)
    keep = np.ones(n, bool)
    keep[at] = False
    assert np.array_equal(got[keep], want[keep])
    # 1 / 2^510 times the densities' sum at most (in the mixed form the difference of a
    # far target and a far source of another leaf is inf - inf in FP32, as ever)
    if form == "PLAIN_FP64":
        assert np.max(np.abs(got[at])) <= np.abs(pts["den"]).sum() * 2.0 ** -510
