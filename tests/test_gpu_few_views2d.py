"""2D calls with few views or few rays, which run the direct kernels, at the
edges of both rules: the values of the line kernels (whose bits they share), of
the oracle, and of a longer scan's first views; fan scans whose rays march over
rows, over columns, over both."""
import importlib

import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _geom(astra, kind, rows, cols, views, start=0.1, total=None):
    n = max(rows, cols)
    ang = (start + np.linspace(0, 2 * np.pi, total or views, endpoint=False)[:views]).astype(np.float32)
    vg = astra.create_vol_geom(rows, cols)
    if kind == 'parallel':
        return astra.create_proj_geom('parallel', 1.0, int(1.4 * n), ang), vg
    return astra.create_proj_geom('fanflat', 1.5, int(1.4 * n), ang, 2.0 * n, 1.0 * n), vg


def _launches():
    return importlib.import_module("astra-toolbox_b200._lib").load().b2t_kernel_launches()


# backprojection: images of one warp a tile (more than 1800 tiles of 32 x 4), of
# fewer, and with more tiles than LINES_BP_WARPS
@pytest.mark.parametrize("kind", ["parallel", "fanflat"])
@pytest.mark.parametrize("n", [476, 484, 680, 700, 1100])
def test_bp_equals_the_views_of_a_longer_scan(astra, orc, kind, n):
    """A scan of few views against the same views with zeros for the rest of a
    longer scan, which is staged; both against the oracle."""
    for views in (1, 2, 8, 9, 12, 13):
        few = astra.Projector2D(*_geom(astra, kind, n, n, views, total=60))
        long_ = astra.Projector2D(*_geom(astra, kind, n, n, 60))
        sino = torch.rand(few.proj_shape, device='cuda')
        full = torch.zeros(long_.proj_shape, device='cuda')
        full[:views] = sino
        a = few.bp(sino, torch.zeros(few.vol_shape, device='cuda'))
        b = long_.bp(full, torch.zeros(few.vol_shape, device='cuda'))
        # the partial sums are cut elsewhere: sums of at most 13 positive terms in
        # two orders, 12 roundings each
        assert bool(((a - b).abs() <= 24 * 2 ** -24 * b).all()), (views, float(((a - b).abs() / b).max()))
        c = few.bp(sino, torch.full_like(a, 0.25), mode=0)
        assert torch.allclose(c, a + 0.25, rtol=1e-6, atol=0)
        if views in (2, 9) and n < 600:
            ref = (orc.fan_bp if kind == 'fanflat' else orc.par_bp)(few.geom.views_array(), sino.cpu().numpy(),
                                                                    few.vol_shape, few.geom.output_scale)
            # positions of up to 350 texels, rounded twice, move by up to 2^-16 texels
            # each, and a sample of this noise by as much as its own size per texel
            assert rel_l2(a.cpu().numpy(), ref) < 2 * 2 ** -16


@pytest.mark.parametrize("kind", ["parallel", "fanflat"])
@pytest.mark.parametrize("rows,cols", [(64, 64), (64, 65), (65, 30), (96, 80), (97, 97), (128, 100), (129, 128)])
def test_fp_against_the_oracle(astra, orc, kind, rows, cols):
    """Launches tell the direct kernel (one) from the lines (two)."""
    for views in (1, 2, 3, 16, 17, 64, 65):
        for start in (0.1, 0.78, 1.6):
            pg, vg = _geom(astra, kind, rows, cols, views, start, total=max(views, 50))
            pr = astra.Projector2D(pg, vg)
            vol = torch.rand(pr.vol_shape, device='cuda')
            n = _launches()
            fp = pr.fp(vol, torch.zeros(pr.proj_shape, device='cuda'))
            n = _launches() - n
            big = max(rows, cols)
            few = views <= 16 and big <= 96 if kind == 'parallel' else views <= 2 and big <= 128 and start == 0.1
            direct = big <= 64 and views <= 64 or few
            assert n == (1 if direct else 2), (views, start, n)
            ref = (orc.fan_fp if kind == 'fanflat' else orc.par_fp)(pr.geom.views_array(), vol.cpu().numpy(),
                                                                    pr.proj_shape[1], pr.geom.output_scale, rays=1)
            assert rel_l2(fp.cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("start", np.linspace(0.0, 1.6, 17))
def test_fan_scans_with_one_set_of_lines(astra, orc, start):
    """Three neighbouring views, whose rays march over rows, over columns or over both,
    with and without supersampling."""
    pg, vg = _geom(astra, 'fanflat', 150, 131, 3, start, total=360)
    for rays in (1, 3):
        pr = astra.Projector2D(pg, vg, {'DetectorSuperSampling': rays})
        vol = torch.rand(pr.vol_shape, device='cuda')
        fp = pr.fp(vol, torch.zeros(pr.proj_shape, device='cuda'))
        ref = orc.fan_fp(pr.geom.views_array(), vol.cpu().numpy(), pr.proj_shape[1], pr.geom.output_scale, rays=rays)
        assert rel_l2(fp.cpu().numpy(), ref) < 1e-5


def test_sirt_of_few_views(astra, orc):
    """SIRT of a large image with few views: the update runs apart from the
    backprojection, with the values of the fused one."""
    pg, vg = _geom(astra, 'parallel', 500, 500, 6)
    sino = torch.rand((6, 700), device='cuda')
    vol = torch.zeros((500, 500), device='cuda')
    ids = [astra.data2d.link('-sino', pg, sino), astra.data2d.link('-vol', vg, vol)]
    cfg = astra.astra_dict('SIRT_CUDA')
    cfg['ProjectionDataId'], cfg['ReconstructionDataId'] = ids
    alg = astra.algorithm.create(cfg)
    astra.algorithm.run(alg, 3)
    pr = astra.Projector2D(pg, vg)
    ones = torch.ones_like(vol)
    lw = pr.fp(ones, torch.zeros_like(sino))
    pw = pr.bp(torch.ones_like(sino), torch.zeros_like(vol))
    inv = lambda w: torch.where(w > 1e-6, 1.0 / w, torch.zeros_like(w))
    x = torch.zeros_like(vol)
    for _ in range(3):
        r = (sino - pr.fp(x, torch.zeros_like(sino))) * inv(lw)
        x = x + pr.bp(r, torch.zeros_like(vol)) * inv(pw)
    # (rays that graze the image have weights of rounding size)
    assert rel_l2(vol.cpu().numpy(), x.cpu().numpy()) < 5e-4
    astra.algorithm.delete(alg)
    for i in ids:
        astra.data2d.delete(i)
