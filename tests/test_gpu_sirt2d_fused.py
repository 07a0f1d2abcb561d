"""SIRT_CUDA's iteration in the projectors' own launches (the residual in the
forward projection, the update in the backprojection) against the same
iteration from separate projections, with bounds and masks; scans of more
views than one backprojection launch holds take the separate update."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views", [7, 61, 1100])
@pytest.mark.parametrize("geom", ["parallel", "fanflat"])
@pytest.mark.parametrize("bounded", [False, True])
@pytest.mark.parametrize("fail", [0, 1])
def test_iterations(astra, views, geom, bounded, fail):
    D = importlib.import_module("astra-toolbox_b200.data2d")
    A = importlib.import_module("astra-toolbox_b200.algorithm")
    lib = importlib.import_module("astra-toolbox_b200._lib").load()
    ang = np.linspace(0, 2 * np.pi, views, endpoint=False).astype(np.float32) + np.float32(0.02)
    vg = astra.create_vol_geom(35, 42)
    pg = astra.create_proj_geom('parallel', 1.0, 61, ang) if geom == 'parallel' else \
        astra.create_proj_geom('fanflat', 1.4, 61, ang, 90.0, 45.0)
    rng = np.random.default_rng(views)
    b = torch.from_numpy(rng.random((views, 61), dtype=np.float32) * 9).cuda()
    x0 = torch.from_numpy(rng.random((35, 42), dtype=np.float32)).cuda()
    lo = torch.full((35, 42), 0.3, device='cuda')
    x = x0.clone()
    ids = [D.link('-sino', pg, b), D.link('-vol', vg, x), D.link('-vol', vg, lo)]
    cfg = astra.astra_dict('SIRT_CUDA')
    cfg['ProjectionDataId'], cfg['ReconstructionDataId'] = ids[:2]
    cfg['option'] = {'Relaxation': 0.9}
    if bounded:
        cfg['option'].update(MinConstraint=0.1, MaxConstraint=0.8, MinMaskId=ids[2])
    a = A.create(cfg)
    A.run(a, 0)  # the weights
    lib.b2t_debug_fail_alloc(fail, None)  # 1: the first projection's scratch fails
    try:
        A.run(a, 3)
    finally:
        lib.b2t_debug_fail_alloc(0, None)
    A.delete(a)
    D.delete(ids)

    pr = astra.Projector2D(pg, vg)
    inv = lambda t: torch.where(t > 1e-6, 1.0 / t, torch.zeros_like(t))  # noqa: E731
    line = inv(pr.fp(torch.ones_like(x0), torch.empty_like(b)))
    pix = inv(pr.bp(torch.ones_like(b), torch.empty_like(x0))) * 0.9
    y = x0.clone()
    for _ in range(3):
        r = (b - pr.fp(y, torch.empty_like(b))) * line
        y = y + pix * pr.bp(r, torch.empty_like(y))
        if bounded:
            y = torch.maximum(y.clamp(0.1, 0.8), lo)
    assert float((x - y).norm()) <= 1e-6 * float(y.norm())
