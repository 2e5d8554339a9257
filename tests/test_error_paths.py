"""Error reporting of the kernels' bounded waits, driven without a fault.

The V list, in both forms, copies each frequency block's translation spectra into
shared memory with a bulk copy and waits on an mbarrier for a bounded number
of tries; when the tries run out the kernel sets the plan's error flag and
returns (after letting the copy land).  kfmm_set_wait_limit(plan, 0) makes
that wait give up at once, so the error path runs on every launch: the solve
must then report KFMM_ERR_CUDA through every call that hands back potentials,
and the next solve with the default limit must succeed with the same
potentials as an untouched plan (the flag is cleared at the start of each
solve).  The reference has no such path: it exits on any CUDA error
(fmm/cuda.cu:19-30).
"""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _setup(K, n=20000, ppb=32, np_=4):
    pts = K.generate_points(n, "uniform", 0, 26)
    tree = K.Tree(pts["sx"], pts["sy"], pts["sz"], pts["tx"], pts["ty"], pts["tz"], ppb)
    return pts, tree


def test_set_wait_limit_rejects_null_plan(K):
    assert K.lib().kfmm_set_wait_limit(None, 0) == 1
    assert K.lib().kfmm_batch_wait(None, None) == 1


FORMS = pytest.mark.parametrize("form", ["MIXED", "PLAIN_FP64"])


@pytest.mark.gpu
@FORMS
def test_wait_timeout_reported_then_cleared(K, cuda_ok, form):
    import torch
    prec = getattr(K, form)
    pts, tree = _setup(K)
    want = K.Plan(tree, 4, prec).evaluate(pts)
    plan = K.Plan(tree, 4, prec)
    plan.set_wait_limit(0)
    with pytest.raises(K.KfmmError, match="bounded wait"):
        plan.evaluate(pts)
    plan.run()
    with pytest.raises(K.KfmmError, match="bounded wait"):
        plan.potentials()
    out = torch.empty(len(want), dtype=torch.float64, device="cuda:0")
    rc = K.lib().kfmm_get_potentials_device(plan.handle, out.data_ptr(), None)
    assert rc == 2 and b"bounded wait" in K.lib().kfmm_last_error()
    plan.set_wait_limit(-1)
    got = plan.evaluate(pts)
    assert np.array_equal(got, want)
    assert K.lib().kfmm_get_potentials_device(plan.handle, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.gpu
@FORMS
def test_batch_wait_reports_timeout(K, cuda_ok, form):
    prec = getattr(K, form)
    pts, tree = _setup(K, n=15000)
    plans = [K.Plan(tree, 4, prec) for _ in range(2)]
    for p in plans:
        p.set_points(pts)
    want = K.Plan(tree, 4, prec).evaluate(pts)
    plans[1].set_wait_limit(0)
    batch = K.Batch(plans, nstreams=2)  # the limit is captured with the launch
    batch.launch()
    with pytest.raises(K.KfmmError, match="solve 1"):
        batch.wait()
    batch.close()
    plans[1].set_wait_limit(-1)
    batch = K.Batch(plans, nstreams=2)
    batch.launch()
    batch.wait()
    for p in plans:
        assert np.array_equal(p.potentials(), want)
    batch.close()


@pytest.mark.gpu
def test_batch_wait_before_a_launch(K, cuda_ok):
    """Nothing was launched, so nothing ran out: a wait reports no error, whatever the
    device memory the batch got held before."""
    import ctypes
    import torch
    torch.cuda.init()
    rt = ctypes.CDLL("libcudart.so.12")  # torch's, already loaded
    pts, tree = _setup(K, n=3000)
    plans = [K.Plan(tree, 4, K.MIXED) for _ in range(40)]
    for p in plans:
        p.set_points(pts)
    torch.cuda.synchronize()
    bufs = [ctypes.c_void_p() for _ in range(8192)]
    for b in bufs:
        assert rt.cudaMalloc(ctypes.byref(b), ctypes.c_size_t(512)) == 0
        assert rt.cudaMemset(b, 1, ctypes.c_size_t(512)) == 0
    assert rt.cudaDeviceSynchronize() == 0
    for b in bufs:
        assert rt.cudaFree(b) == 0
    batch = K.Batch(plans, nstreams=2)
    batch.wait()
    batch.launch()
    batch.wait()
    batch.close()


# The first plan of the process lives in a context of its own, which ends while a plan
# of the device's primary context is in use (as when one of two devices is reset).
ENDED_CONTEXT = """
import ctypes
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import __graft_entry__
K = __graft_entry__.load_package()
pts = K.generate_points(5000, "uniform", 0, 26)
tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], 32)
cu = ctypes.CDLL("libcuda.so.1")
def ok(rc):
    assert rc == 0, rc
dev, ctx = ctypes.c_int(), ctypes.c_void_p()
ok(cu.cuInit(0))
ok(cu.cuDeviceGet(ctypes.byref(dev), 0))
ok(cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, dev))
first = K.Plan(tree, 4, K.MIXED)
want = first.evaluate(pts)
ok(cu.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p())))
plan = K.Plan(tree, 4, K.MIXED)
assert np.array_equal(plan.evaluate(pts), want)
ok(cu.cuCtxPushCurrent_v2(ctx))
first.close()
ok(cu.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p())))
ok(cu.cuCtxDestroy_v2(ctx))
assert np.array_equal(plan.evaluate(pts), want)
later = K.Plan(tree, 4, K.MIXED)
for p in (later, plan):
    p.set_wait_limit(0)
    try:
        p.evaluate(pts)
        raise SystemExit("the flag did not arrive")
    except K.KfmmError as e:
        assert "bounded wait" in str(e)
    p.set_wait_limit(-1)
    assert np.array_equal(p.evaluate(pts), want)
print("done")
"""


@pytest.mark.gpu
def test_flags_outlive_the_first_plans_context(cuda_ok):
    r = subprocess.run([sys.executable, "-c", ENDED_CONTEXT, ROOT], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr
