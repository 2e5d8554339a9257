"""Leaves of millions of targets: a tree splits on its sources only, so few sources
and many targets leave one leaf.  Its job bounds pass 32 bits when they are formed
as rows x parts (from 2,965,761 targets at 4 rows a job, 1,482,881 at 1).
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "kifmm--hybrid--double-only_b200", "csrc")


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    """The job split of csrc/host.h, compiled by itself."""
    d = tmp_path_factory.mktemp("split")
    src, lib = d / "split.cc", d / "split.so"
    src.write_text('#include "host.h"\n'
                   'extern "C" int parts(int n, int r) { return kfmm::even_parts(n, r); }\n'
                   'extern "C" int begin(int n, int r, int c) {\n'
                   '  return kfmm::even_part_begin(n, r, c);\n}\n')
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC,
                           "-I", os.path.join(ROOT, "include"), str(src), "-o", str(lib)])
    return ctypes.CDLL(str(lib))


@pytest.mark.parametrize("rows", [1, 4, 6])
@pytest.mark.parametrize("count", [0, 1, 31, 32, 33, 128, 129, 421, 1482880, 1482881, 2965760,
                                   2965761, 3100000, 40000000])
def test_split_covers_every_target_once(split, count, rows):
    parts = split.parts(count, rows)
    assert parts == -(-(-(-count // 32)) // rows)
    step = max(1, parts // 5000)  # the large ones in strides, with both ends
    for c in sorted(set(range(0, parts, step)) | set(range(max(0, parts - 50), parts))):
        lo, hi = split.begin(count, rows, c), split.begin(count, rows, c + 1)
        full = -(-count // 32)
        assert lo == 32 * (full * c // parts) and hi == min(count, 32 * (full * (c + 1) // parts))
        assert 0 < hi - lo <= 32 * rows
    ends = split.begin(count, rows, 0), split.begin(count, rows, parts)
    assert parts == 0 or ends == (0, count)


def _leaf(nt):
    rng = np.random.default_rng(nt)
    pts = {k: rng.uniform(-1, 1, 8) for k in ("sx", "sy", "sz")}
    pts["den"] = rng.uniform(0.1, 1, 8)
    pts.update({k: rng.uniform(-1, 1, nt) for k in ("tx", "ty", "tz")})
    return pts


def _reference(pts):
    """The direct sum and the closest pair."""
    out, near = np.zeros(len(pts["tx"])), np.inf
    for j in range(8):
        r = np.sqrt(sum((pts["t" + c] - pts["s" + c][j]) ** 2 for c in "xyz"))
        near = min(near, r.min())
        out += pts["den"][j] / r
    return out / (4 * np.pi), near


def _check(got, ref, near, mixed):
    """Eight positive terms in FP64: 8 eps of order and 8 of the terms; mixed: FP32
    coordinates put a pair at distance r off by about 2^-24 / r."""
    tol = 8 * 2.0 ** -24 * (1 + 1 / near) if mixed else 16 * 2.0 ** -52
    assert np.max(np.abs(got - ref) / ref) <= tol


def _tree(K, pts):
    tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], 64, device=True)
    assert tree.desc.num_nodes == 1
    return tree


@pytest.mark.gpu
@pytest.mark.parametrize("precision,nt,tuning", [("plain", 3100000, None),
                                                 ("plain", 1600000, {"job_rows": 1}),
                                                 ("mixed", 2000000, {"job_rows": 1}),
                                                 ("mixed", 3100000, None)])
def test_one_large_leaf(K, cuda_ok, precision, nt, tuning):
    mixed = precision == "mixed"
    pts = _leaf(nt)
    tree = _tree(K, pts)
    plan = K.Plan(tree, 4, K.MIXED if mixed else K.PLAIN_FP64, tuning=tuning)
    _check(plan.evaluate(pts), *_reference(pts), mixed)


@pytest.mark.gpu
@pytest.mark.parametrize("tuning", [None, {"job_rows": 1}])
def test_large_leaves_in_a_batch(K, cuda_ok, tuning):
    cases = [_leaf(3100000), _leaf(3000001)]
    plans = [K.Plan(_tree(K, p), 4, K.PLAIN_FP64, tuning=tuning) for p in cases]
    for plan, pts in zip(plans, cases):
        plan.set_points(pts)
    batch = K.Batch(plans, nstreams=2)
    batch.launch()
    batch.wait()
    for plan, pts in zip(plans, cases):
        _check(plan.potentials(), *_reference(pts), False)
    batch.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["PLAIN_FP64", "MIXED"])
def test_plan_memory_per_target(K, cuda_ok, form):
    """A target costs 72 bytes of a plan: 24 of upload staging, 32 in leaf order, 8 of
    permutations, 8 of potential.  Device memory comes in pages of 2 MiB, which rounds
    these seven arrays up by 14 MiB at most; the rest of this plan (jobs 1.4 MB,
    operators 3 MB, eight sources) takes five such pages at most.  Another 8 bytes
    a target would be 30 MiB."""
    import torch
    prec = getattr(K, form)
    small = K.generate_points(2000, "uniform", 0, 1)
    tree = K.Tree(*[small[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], 64)
    K.Plan(tree, 4, prec).evaluate(small)  # modules loaded, flag slots allocated
    nt = 4000000
    pts = _leaf(nt)
    tree = _tree(K, pts)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    plan = K.Plan(tree, 4, prec)
    used = free - torch.cuda.mem_get_info()[0]
    assert used <= 72 * nt + (24 << 20), used / nt
    plan.set_points(pts)
    plan.run()
    got, leaf = plan.potentials(), plan.read(3, nt)
    assert np.array_equal(leaf, got[tree.array("trg_perm")])
    assert plan.read(3, 5).tolist() == leaf[:5].tolist()
