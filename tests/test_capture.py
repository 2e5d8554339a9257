"""kfmm_run captured into a CUDA graph by the caller (GPU): the far field's
programmatic launches become graph edges, and replays give the direct run's bits."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("dist,n,ppb,np_", [("uniform", 20000, 64, 4),
                                            ("ellipseUniformAngles", 9000, 24, 3)])
def test_caller_capture_replays(K, cuda_ok, precision, dist, n, ppb, np_):
    import torch
    pts = K.generate_points(n, dist, 0, 4)
    tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], ppb)
    plan = K.Plan(tree, np_, K.PLAIN_FP64 if precision == "plain" else K.MIXED)
    want = plan.evaluate(pts)
    other = {**pts, "den": 1.0 - pts["den"]}
    want_other = plan.evaluate(other)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run(torch.cuda.current_stream().cuda_stream)
    for p, w in ((pts, want), (other, want_other), (pts, want)):
        plan.set_points(p)
        torch.cuda.synchronize()
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(plan.potentials(), w)


@pytest.mark.gpu
def test_back_to_back_runs(K, cuda_ok):
    """Runs queued without waiting, on a stream of their own and on the default
    stream, densities changing between them."""
    import torch
    n = 6000
    pts = K.generate_points(n, "ellipsoidSurface", 0, 8)
    tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], 20)
    dens = [pts["den"], 1.0 - pts["den"], 0.5 * pts["den"]]
    for precision in (K.PLAIN_FP64, K.MIXED):
        plan = K.Plan(tree, 4, precision)
        want = [plan.evaluate({**pts, "den": d}) for d in dens]
        src = [torch.from_numpy(pts[k]).cuda() for k in ("sx", "sy", "sz")]
        dd = [torch.from_numpy(np.ascontiguousarray(d)).cuda() for d in dens]
        out = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in dens]
        torch.cuda.synchronize()
        for stream in (torch.cuda.Stream().cuda_stream, None):
            for rep in range(5):
                for d, o in zip(dd, out):
                    K.check(K.lib().kfmm_set_sources_device(
                        plan.handle, *[t.data_ptr() for t in src], d.data_ptr(), stream), "sources")
                    for _ in range(2):
                        plan.run(stream)
                    K.check(K.lib().kfmm_get_potentials_device(plan.handle, o.data_ptr(), stream),
                            "potentials")
            for o, w in zip(out, want):
                assert np.array_equal(o.cpu().numpy(), w)
