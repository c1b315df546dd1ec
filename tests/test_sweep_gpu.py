"""The batched lens-parameter sweep (one persistent launch over many samples of uneven size,
KB widths 6 and 8 side by side): against the per-sample entry points (themselves pinned to the
oracle) and, for a few samples, against the oracle directly."""
import numpy as np
import pytest
import torch

import oracle as O
from helpers import REL_L2_FP32

pytestmark = pytest.mark.gpu


def _samples(rng, k=10):
    from lentils_gb300.sweep import draw_samples
    s = draw_samples(rng, k, sizes=(32, 48, 64), nvis_range=(2000, 20000), eps=0.01)
    # accuracy targets on both sides of the KB-width threshold
    for i, x in enumerate(s):
        x.tol = 1e-4 if i % 2 else 1e-6
        x.pix = 0.04
    return s


@pytest.fixture(scope="module")
def sweep(tmp_path_factory):
    from lentils_gb300.autotune import Autotuner
    from lentils_gb300.sweep import BatchedSweep
    path = str(tmp_path_factory.mktemp("tune") / "cache.json")
    tuner = Autotuner(path=path, tiles=(8, 16), chunks=(256, 1024), reps=1, mode="batched")
    sw = BatchedSweep(_samples(np.random.default_rng(11)), tuner=tuner)
    tuner.save()
    return sw, tuner, path


def test_sweep_mixes_widths_and_tunes(sweep):
    from lentils_gb300.autotune import Autotuner
    sw, tuner, path = sweep
    widths = {s.info["w2"] for s in sw.samples}
    assert widths == {6, 8}
    assert tuner.tuned > 0
    again = Autotuner(path=path, tiles=(8, 16), chunks=(256, 1024), mode="batched")
    for s in sw.samples:
        p = sw.plans[sw.samples.index(s)]
        assert again.params(p.nu, p.nv, 0, 0, s.info["w2"], s.nvis) == (s.info["tile"],
                                                                        s.info["chunk"])
    assert again.tuned == 0
    st = sw.stats()
    assert st["nsamples"] == len(sw.samples) and st["nwork"] > 0 and st["blocks"] > 0


@pytest.mark.parametrize("use_graph", [True, False])
def test_sweep_matches_per_sample_entry_points(sweep, use_graph):
    from lentils_gb300.lens_models import GlobalLensModel
    sw, _, _ = sweep
    for go in sw.grid_out:
        go.fill_(float("nan"))
    sw.run(use_graph=use_graph)
    sw.run(use_graph=use_graph)  # a second run overwrites (grids are cleared per run)
    sw.stream.synchronize()
    for k, s in enumerate(sw.samples):
        plan = sw.plans[k]
        v_ref = plan.degrid(sw.grid_in[k])
        assert torch.equal(sw.vis_out[k], v_ref), k
        g_ref = plan.grid(sw.vis_in[k])
        rel = float((sw.grid_out[k] - g_ref).abs().norm() / g_ref.abs().norm())
        assert rel < 1e-6, (k, rel)
        pts = torch.as_tensor(sw.pixel_points(k)).cuda()
        b_ref = GlobalLensModel(s.lenses).deflect(pts, 2.0).float()
        assert torch.allclose(sw.beta_out[k], b_ref, rtol=0, atol=2e-6), k


@pytest.mark.parametrize("form", [1, 2])
def test_sweep_kernel_forms(sweep, form):
    """The other item forms of the sweep kernel (column-pair gridder; same-cell chunk or
    per-visibility degridding) on the same samples, plans and inputs: visibilities identical,
    grids within FP32 summation order, deflections identical."""
    from lentils_gb300.autotune import Autotuner
    from lentils_gb300.sweep import BatchedSweep
    sw, _, path = sweep
    sw.run(use_graph=True)
    sw.stream.synchronize()
    tuner = Autotuner(path=path, tiles=(8, 16), chunks=(256, 1024), mode="batched")
    other = BatchedSweep(_samples(np.random.default_rng(11)), tuner=tuner, form=form)
    assert tuner.tuned == 0
    other.run(use_graph=True)
    other.stream.synchronize()
    for k in range(len(sw.samples)):
        assert torch.equal(other.grid_in[k], sw.grid_in[k]) and torch.equal(other.vis_in[k], sw.vis_in[k])
        assert torch.equal(other.vis_out[k], sw.vis_out[k]), k
        rel = float((other.grid_out[k] - sw.grid_out[k]).abs().norm() / sw.grid_out[k].abs().norm())
        assert rel < 1e-6, (k, rel)
        assert torch.equal(other.beta_out[k], sw.beta_out[k]), k


@pytest.mark.parametrize("nbeta,sizes", [(1, (33, 20)), (4, (40, 64)), (6, (48, 50))])
def test_tables_and_odd_grids(nbeta, sizes):
    """Plans with one, four (the most that get kernels of their own) and six different
    Kaiser-Bessel tables in one sweep, grids of odd size, a sample without visibilities and one
    without pixels, output grids 8 bytes off a 16-byte boundary; on the stream and as a graph."""
    import ctypes
    from lentils_gb300 import _native as N
    from lentils_gb300.gridding import GriddingPlan
    from lentils_gb300.lens_models import ExternalPotential, GlobalLensModel
    rng = np.random.default_rng(nbeta)
    lens = GlobalLensModel([ExternalPotential(z=0.5, x=0.0, y=0.0, ss=0.05, sa=20.0)])
    la = lens.setup_raytracing(2.0)
    cs, keep = (N.SweepSampleC * (nbeta + 2))(), []
    for k in range(nbeta + 2):
        w = 3 if k % 2 else 4
        four = O.FourierGeom(O.ImageGeom((sizes[k % 2] * 2 + k % 3, sizes[1] * 2 + 1),
                                         [(-1.0, 1.0), (-1.0, 1.0)]))
        n = 0 if k == nbeta else 700 + 300 * k
        uvw = O.synth_uv(rng, n, four, 0.4, w) if n else np.zeros((0, 3))
        beta = 2.34 * 2 * w * (1 + 0.01 * (k % nbeta))
        plan = GriddingPlan(uvw, [1.0], four.nu, four.nv, four.du, four.dv, 0.0, 0.0, w, beta,
                            tile=8 if k % 2 else 16, chunk=256)
        gi = torch.randn((four.nu, four.half_nv), dtype=torch.complex64, device="cuda")
        vi = torch.randn(max(1, n), dtype=torch.complex64, device="cuda")
        go = torch.full((four.nu * four.half_nv + 1,), float("nan"), dtype=torch.complex64,
                        device="cuda")[k % 2:][:four.nu * four.half_nv]
        vo = torch.empty_like(vi)
        nx = 0 if k == nbeta + 1 else 50 + k
        bo = torch.empty((max(1, nx * nx), 2), dtype=torch.float32, device="cuda")
        c = cs[k]
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())
        c.plan, c.grid_in, c.vis_out, c.vis_in = plan.handle, ptr(gi), ptr(vo), ptr(vi)
        c.grid_out, c.lenses, c.nlenses = ptr(go), ctypes.c_void_p(la.ctypes.data), len(la)
        c.nx = c.ny = nx
        c.x0 = c.y0 = -1.0
        c.dx = c.dy = 0.04
        c.beta_out = ptr(bo)
        keep.append((plan, gi, vi, go, vo, bo, n, nx))
    h = ctypes.c_void_p()
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    sp = ctypes.c_void_p(st.cuda_stream)
    N.check(N.lib().lentils_sweep_create(ctypes.byref(h), cs, nbeta + 2, 0, sp))
    try:
        for graph in (0, 1, 1):
            for _, _, _, go, vo, bo, _, _ in keep:
                go.fill_(float("nan"))
                vo.zero_()
                bo.zero_()
            torch.cuda.synchronize()
            N.check(N.lib().lentils_sweep_run(h, graph, sp))
            st.synchronize()
            for plan, gi, vi, go, vo, bo, n, nx in keep:
                ref = plan.grid(vi[:n])
                err = (go.reshape(ref.shape) - ref).abs().norm()
                assert float(err) <= 1e-6 * float(ref.abs().norm())
                if n:
                    assert torch.equal(vo, plan.degrid(gi))
                if nx:
                    c = -1.0 + 0.04 * np.arange(nx)
                    pts = np.stack(np.meshgrid(c, c, indexing="ij"), -1).reshape(-1, 2)
                    b = lens.deflect(pts, 2.0)
                    assert np.max(np.abs(bo.cpu().numpy() - b)) < 2e-6
    finally:
        N.lib().lentils_sweep_destroy(h)


def test_sweep_against_oracle(sweep):
    """Two samples (one per KB width) in user row order against the FP64 CPU oracle."""
    from lentils_gb300.lens_models import GlobalLensModel
    sw, _, _ = sweep
    rng = np.random.default_rng(3)
    ks = [0, 1]
    ys = {}
    for k in ks:
        plan = sw.plans[k]
        y = O.complex_normal(rng, plan.nvis)
        sw.vis_in[k].copy_(plan.to_plan(torch.as_tensor(y).cuda()))
        ys[k] = y
    sw.run()
    sw.stream.synchronize()
    for k in ks:
        s, plan = sw.samples[k], sw.plans[k]
        four = O.FourierGeom.__new__(O.FourierGeom)
        four.nu, four.nv, four.half_nv = plan.nu, plan.nv, plan.half_nv
        four.du, four.dv = plan.du, plan.dv
        four.gcx = four.gcy = 0.0
        four._chan = np.zeros(1)
        vis = O.VisGeom(sw.uvw[k], [1.0])
        w, beta = plan.wsup, plan.kb_beta
        g_in = sw.grid_in[k].cpu().numpy().astype(np.complex128)
        v_or = O.degrid(vis, four, g_in, w, beta)
        v_us = plan.from_plan(sw.vis_out[k]).cpu().numpy()
        assert O.rel_l2(v_us, v_or) < REL_L2_FP32
        g_or = O.grid(vis, four, ys[k], w, beta)
        assert O.rel_l2(sw.grid_out[k].cpu().numpy(), g_or) < REL_L2_FP32
        lenses = GlobalLensModel(s.lenses).setup_raytracing(2.0)
        b_or = O.deflect(lenses, sw.pixel_points(k))
        assert np.max(np.abs(sw.beta_out[k].cpu().numpy() - b_or)) < 2e-6


def test_single_plan_tuning(tmp_path):
    """Single-plan mode: every (tile, chunk) candidate timed on its own plan; the cache
    answers the same class without tuning again."""
    from lentils_gb300.autotune import Autotuner
    path = str(tmp_path / "single.json")
    t = Autotuner(path=path, tiles=(8, 16), chunks=(256, 1024), reps=1)
    p = t.params(128, 128, 2e4, 2e4, 8, 5000)
    assert p in {(8, 256), (8, 1024), (16, 256), (16, 1024)} and t.tuned == 1
    assert len(t.cache[t.key(128, 128, 8, 5000)]["candidates"]) == 4
    t.save()
    assert Autotuner(path=path).params(128, 128, 0, 0, 8, 5000) == p

