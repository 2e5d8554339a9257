"""Batched solves under one CUDA graph (kfmm_batch_*), with leaf sizes and
launch choices from the autotuner: a smaller instance of the batched
workload (solves of uneven size, uniform cube and ellipsoid surface, NP 3 and
4, mixed form).

* every solve's potentials from the graph replay equal, bit for bit, those of
  the same plan run on its own (the kernels are deterministic), on two
  launches in a row;
* every solve's relative L2 error against an exact direct sum on sampled
  targets is at most 2x the plain FP64 form's error for the same tree.
"""
import numpy as np
import pytest


@pytest.mark.gpu
def test_batched_graph_matches_single_runs(K, oracle_mod, cuda_ok, tmp_path):
    from kifmm_b200 import autotune, batched
    table = autotune.ConfigTable(str(tmp_path / "configs.json"),
                                 knobs=(("job_rows", (0, 4)), ("nf_blocks", (0, 5))),
                                 candidates=(16, 32, 64))
    sp = batched.specs(12, nmin=4096, nmax=40000, seed=7)
    B = batched.BatchedSolves(K, sp, K.MIXED, table=table, nstreams=4, num_check=60)
    single = []
    for s in B.solves:
        s["plan"].run()
        single.append(s["plan"].potentials())
    for rep in range(2):
        B.launch()
        got = B.potentials()
        for i, (a, b) in enumerate(zip(got, single)):
            assert np.array_equal(a, b), f"solve {i} launch {rep}"
    for s, pot in zip(B.solves, single):
        pts = s["pts"]
        plain = K.Plan(s["tree"], s["np"], K.PLAIN_FP64).evaluate(pts)
        ids = pts["check_ids"]
        d = oracle_mod.direct(pts["tx"][ids], pts["ty"][ids], pts["tz"][ids], pts["sx"], pts["sy"],
                              pts["sz"], pts["den"])
        e_mixed = np.linalg.norm(pot[ids] - d) / np.linalg.norm(d)
        e_plain = np.linalg.norm(plain[ids] - d) / np.linalg.norm(d)
        print(f"{s['distribution']} n={s['n']} np={s['np']} ppb={s['ppb']}: mixed {e_mixed:.3e} "
              f"plain {e_plain:.3e}")
        assert e_mixed <= 2.0 * e_plain
    assert (tmp_path / "configs.json").exists()
    assert any(s["tuning"] is not None for s in B.solves)
    B.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["PLAIN_FP64", "MIXED"])
@pytest.mark.parametrize("tuning", [None, {"job_rows": 2}])
def test_batch_of_either_form_and_job_kind(K, cuda_ok, form, tuning):
    """Batches whose near fields are team jobs (plain plans), and team jobs beside
    one-warp jobs (a mixed plan of more target leaves than four times the device's
    warps, between two small ones), bit for bit the single runs."""
    import torch
    prec = getattr(K, form)
    plans, want = [], []
    for n, dist, ppb, np_ in ((20000, "uniform", 40, 4), (400000, "uniform", 12, 3),
                              (9000, "ellipsoidSurface", 24, 3)):
        pts = K.generate_points(n, dist, 0, n)
        tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], ppb)
        leaves = np.count_nonzero((tree.array("child") == -1) & (tree.array("trg_num") > 0))
        warps = 64 * torch.cuda.get_device_properties(0).multi_processor_count
        assert (leaves > 4 * warps) == (n == 400000)
        plans.append(K.Plan(tree, np_, prec, tuning=tuning))
        want.append(plans[-1].evaluate(pts))
    batch = K.Batch(plans, nstreams=2)
    for _ in range(2):
        batch.launch()
        batch.wait()
        for plan, w in zip(plans, want):
            assert np.array_equal(plan.potentials(), w)
    batch.close()


def test_batch_rejects_bad_arguments(K):
    import ctypes
    h = ctypes.c_void_p()
    arr = (ctypes.c_void_p * 1)(None)
    assert K.lib().kfmm_batch_create(arr, 1, 1, ctypes.byref(h)) != 0
    assert K.lib().kfmm_batch_create(arr, 0, 1, ctypes.byref(h)) != 0
    assert K.lib().kfmm_batch_launch(None, None) != 0


def test_specs_follow_the_batched_workload():
    from kifmm_b200 import batched
    sp = batched.specs(256)
    ns = np.array([s["n"] for s in sp])
    assert ns.min() >= 4096 and ns.max() <= 262144
    assert sum(s["distribution"] == "uniform" for s in sp) == 128
    assert {s["np"] for s in sp} == {3, 4}
