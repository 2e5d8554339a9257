"""The autotuner (leaf size, then the kernels' launch choices by coordinate
descent) on a small surface cloud, and the table it ships for the batched
workload."""
import json
import os

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TABLE = os.path.join(ROOT, "kifmm--hybrid--double-only_b200", "tuning_data",
                     "b200_batched_configs.json")


@pytest.mark.skipif(not os.path.exists(TABLE), reason="no tuning table")
def test_shipped_table_covers_the_batched_workload(K):
    from kifmm_b200 import autotune, batched
    with open(TABLE) as f:
        picks = json.load(f)
    fields = {n for n, _ in autotune.KNOBS}
    for prec in (K.MIXED, K.PLAIN_FP64):
        for sp in batched.specs(256):
            e = picks[autotune.ConfigTable.key(sp["distribution"], sp["n"], sp["np"], prec)]
            assert e["ppb"] in (32, 64, 128, 256)
            assert set(e["tuning"]) <= fields
            if prec != K.MIXED:
                assert not set(e["tuning"]) & set(autotune.MIXED_ONLY)


@pytest.mark.gpu
def test_tune_keeps_the_fastest_measured_config(K, cuda_ok):
    from kifmm_b200 import autotune
    pts = K.generate_points(60000, "ellipsoidSurface", 0, 3)
    knobs = (("job_rows", (0, 4)), ("nf_blocks", (0, 5, 6)), ("splitk_max", (0, 1)))
    r = autotune.tune(K, pts, 4, K.MIXED, candidates=(32, 64, 128), knobs=knobs)
    assert r["ppb"] in (32, 64, 128)
    measured = list(r["sweep"]["leaf"].values())
    for d in r["sweep"]["knobs"].values():
        measured += list(d.values())
    assert r["ms"] <= min(measured) * (1 + autotune.KEEP_GAIN) + 1e-9
    # launch choices other than the split-K factor do not change the
    # arithmetic: the tuned plan gives the automatic plan's potentials
    tree = K.Tree(pts["sx"], pts["sy"], pts["sz"], pts["tx"], pts["ty"], pts["tz"], r["ppb"])
    tun = {k: v for k, v in r["tuning"].items() if k != "splitk_max"}
    a = K.Plan(tree, 4, K.MIXED).evaluate(pts)
    b = K.Plan(tree, 4, K.MIXED, tuning=tun).evaluate(pts)
    assert np.array_equal(a, b)
    print(f"tuned: ppb {r['ppb']} {r['tuning']} {r['ms']:.3f} ms; sweep {r['sweep']}")


def test_plan_rejects_bad_tuning(K):
    pts = K.generate_points(2000, "uniform", 0, 1)
    tree = K.Tree(pts["sx"], pts["sy"], pts["sz"], pts["tx"], pts["ty"], pts["tz"], 32)
    for bad in ({"nf_blocks": 3}, {"job_rows": 7}, {"had_windows": 9}, {"splitk_max": -1}):
        with pytest.raises(K.KfmmError, match="tuning value out of range"):
            K.Plan(tree, 4, K.MIXED, tuning=bad)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["plain", "mixed"])
def test_set_tuning_in_place(K, cuda_ok, precision):
    """Re-chunked near-field jobs, other resident-block counts and Hadamard
    shapes give the same potentials bit for bit; a different split-K factor
    reorders the level products' sums only: FP64 rounding, amplified by the
    pseudo-inverses' condition number, which the mixed form's FP32 rounding
    of spectra and sources then shows at its own level (~1e-7)."""
    prec = K.PLAIN_FP64 if precision == "plain" else K.MIXED
    pts = K.generate_points(50000, "uniform", 0, 9)
    tree = K.Tree(pts["sx"], pts["sy"], pts["sz"], pts["tx"], pts["ty"], pts["tz"], 64)
    want = K.Plan(tree, 6, prec).evaluate(pts)
    plan = K.Plan(tree, 6, prec)
    for cfg in ({"job_rows": 3}, {"job_rows": 1, "nf_blocks": 5, "had_windows": 2}, None):
        plan.set_tuning(cfg)
        assert np.array_equal(plan.evaluate(pts), want), cfg
    plan.set_tuning({"splitk_max": 1})
    got = plan.evaluate(pts)
    tol = 1e-9 if precision == "plain" else 1e-6
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < tol


def _many_leaves(K, seed=9):
    """A cloud whose mixed near field runs one warp per job on any device of this
    size: more target leaves than four times the warps that its SMs can hold."""
    import torch
    pts = K.generate_points(400000, "uniform", 0, seed)
    tree = K.Tree(pts["sx"], pts["sy"], pts["sz"], pts["tx"], pts["ty"], pts["tz"], 12)
    leaves = np.count_nonzero((tree.array("child") == -1) & (tree.array("trg_num") > 0))
    assert leaves > 4 * 64 * torch.cuda.get_device_properties(0).multi_processor_count
    return pts, tree


@pytest.mark.gpu
def test_set_tuning_of_one_warp_jobs(K, cuda_ok):
    """The same for the one-warp near field, whose jobs job_rows re-chunks and whose
    kernel nf_blocks chooses (the clouds above are small enough for team jobs)."""
    pts, tree = _many_leaves(K)
    plan = K.Plan(tree, 3, K.MIXED)
    want = plan.evaluate(pts)
    for cfg in ({"job_rows": 1}, {"job_rows": 3, "nf_blocks": 5}, {"job_rows": 6, "nf_blocks": 6},
                {"nf_blocks": 5}, None):
        plan.set_tuning(cfg)
        assert np.array_equal(plan.evaluate(pts), want), cfg
    plain = K.Plan(tree, 3, K.PLAIN_FP64).evaluate(pts)
    # FP32 coordinates and pair terms, as on every uniform cloud
    assert np.linalg.norm(want - plain) / np.linalg.norm(plain) < 1e-6


@pytest.mark.gpu
def test_one_warp_leaf_of_several_rows(K, cuda_ok):
    """One-warp jobs of 1 to 6 rows: a single leaf of many targets (its 16,000 jobs are
    more than four for each of the 24 x 148 warps that the kernel keeps resident)."""
    rng = np.random.default_rng(4)
    nt = 3000000 + 77
    pts = {k: rng.uniform(-1, 1, 100) for k in ("sx", "sy", "sz")}
    pts["den"] = rng.uniform(0, 1, 100)
    pts.update({k: rng.uniform(-1, 1, nt) for k in ("tx", "ty", "tz")})
    tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], 100, device=True)
    plan = K.Plan(tree, 4, K.MIXED)
    want = plan.evaluate(pts)
    for rows in range(1, 7):
        plan.set_tuning({"job_rows": rows})
        assert np.array_equal(plan.evaluate(pts), want), rows
