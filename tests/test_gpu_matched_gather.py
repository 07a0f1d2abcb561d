"""The exact adjoint gathered per voxel (B2T_MATCHED_PATH=gather: at any size) against the FP64 transpose and the
scattered adjoint (B2T_MATCHED_PLAIN=1): volumes around the 8 x 8 x 64 and 16 x 16 x 64 tiles,
detectors of every row spacing from 1/4 texel on, detector columns that
run either way, off-centre and cropped detectors, split views, storage types,
ADD mode, row pitches; views that the gather does not take are scattered."""
import ctypes
import importlib

import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _scatters():
    out = (ctypes.c_uint64 * 4)()
    assert importlib.import_module("astra-toolbox_b200._lib").load().b2t_matched_path_stats(out) == 0
    return out[2] + out[3]


def _vec(kind, n, pu, pv, flip=False, shift=(0.0, 0.0), so=150.0, od=60.0):
    out = np.zeros((n, 12))
    for i in range(n):
        t = 2 * np.pi * i / n + 0.07
        u, v = np.array([np.cos(t), np.sin(t), 0.0]), np.array([0.0, 0.0, 1.0])
        ray = np.array([-np.sin(t), np.cos(t), 0.0])
        c = ray * od + shift[0] * u + shift[1] * v
        out[i] = np.concatenate([-ray * so if kind == 'cone_vec' else ray, c, pu * (-u if flip else u), pv * v])
    return out


def _check(astra, orc, pg, vg, monkeypatch, gathered=True, dtype="float32", keep=1.0):
    pr = astra.Projector3D(pg, vg, {'ProjectionKernel': 'matched_bp'})
    proj = np.random.default_rng(pr.vol_shape[0]).standard_normal(pr.proj_shape).astype(np.float32)
    proj *= np.random.default_rng(1).random((1,) + pr.proj_shape[1:]) < keep
    tp = torch.from_numpy(proj).cuda().to(getattr(torch, dtype))
    monkeypatch.setenv("B2T_MATCHED_PATH", "gather")
    _scatters()
    a = torch.zeros(pr.vol_shape, device='cuda', dtype=tp.dtype)
    pr.bp(tp, a)
    n = _scatters()
    assert gathered is None or (n == 0) == gathered
    monkeypatch.setenv("B2T_MATCHED_PLAIN", "1")
    b = torch.zeros_like(a)
    pr.bp(tp, b)
    monkeypatch.delenv("B2T_MATCHED_PLAIN")
    assert _scatters() > 0
    ref = orc.fp3d_transpose(pr.geom.kind, pr.geom.views_array(), tp.float().cpu().numpy(), pr.vol_shape,
                             pr.geom.vol_scale)
    # one rounding of the output in 16 bits, FP32 sums in another order else
    tol = {"float32": 1e-5, "float16": 1e-3, "bfloat16": 8e-3}[dtype]
    assert rel_l2(a.float().cpu().numpy(), ref) < tol
    assert rel_l2(a.float().cpu().numpy(), b.float().cpu().numpy()) < tol
    c = a.clone()
    pr.bp(tp, c, mode=0)
    assert rel_l2(c.float().cpu().numpy(), 2 * ref) < tol


@pytest.mark.parametrize("shape", [(1, 1, 1), (63, 15, 17), (64, 16, 16), (65, 17, 15), (33, 50, 31), (130, 20, 40)])
@pytest.mark.parametrize("kind", ["cone_vec", "parallel3d_vec"])
def test_tile_edges(astra, orc, shape, kind, monkeypatch):
    nz, ny, nx = shape
    vg = astra.create_vol_geom(ny, nx, nz)
    for n, flip in ((3, False), (17, True), (50, False)):
        pg = astra.create_proj_geom(kind, 67, 75, _vec(kind, n, 1.0, 0.95, flip))
        _check(astra, orc, pg, vg, monkeypatch)


@pytest.mark.parametrize("pv", [0.45, 0.55, 0.75, 0.9, 1.2, 2.9])
def test_row_spacings(astra, orc, pv, monkeypatch):
    vg = astra.create_vol_geom(24, 30, 40)
    for pu in (0.3, 1.0, 3.0):
        for kind in ("cone_vec", "parallel3d_vec"):
            pg = astra.create_proj_geom(kind, 41, 53, _vec(kind, 20, pu, pv, shift=(3.3, -2.7)))
            # (edge columns of wide detectors have rows below a quarter of a texel
            # apart at the finest; rows of more than 1 are scattered)
            _check(astra, orc, pg, vg, monkeypatch, gathered=None if pv < 0.6 else pv * (150 / 210 if kind == "cone_vec" else 1) < 1.0)


@pytest.mark.parametrize("keep", [0.0, 0.02, 0.3, 0.9])
def test_zero_columns(astra, orc, keep, monkeypatch):
    vg = astra.create_vol_geom(24, 40, 33)
    for pu in (0.3, 1.0, 2.5):
        pg = astra.create_proj_geom('cone_vec', 41, 70, _vec('cone_vec', 20, pu, 1.0))
        _check(astra, orc, pg, vg, monkeypatch, keep=keep)


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_storage(astra, orc, dtype, monkeypatch):
    vg = astra.create_vol_geom(40, 36, 70, -20, 16, -22.0, 18.0, -30.0, 40.0)
    pg = astra.create_proj_geom('cone', 1.1, 0.9, 60, 64, np.linspace(0, 2 * np.pi, 30, endpoint=False), 150.0, 60.0)
    _check(astra, orc, pg, vg, monkeypatch, dtype=dtype)


def test_anisotropic_voxels(astra, orc, monkeypatch):
    vg = astra.create_vol_geom(40, 36, 30, -18, 18, -30.0, 30.0, -18.0, 18.0)
    pg = astra.create_proj_geom('cone', 1.1, 0.9, 60, 64, np.linspace(0, 2 * np.pi, 30, endpoint=False), 150.0, 60.0)
    _check(astra, orc, pg, vg, monkeypatch)


@pytest.mark.parametrize("case", ["fine", "flipped_rows", "tilted"])
def test_scattered_views(astra, orc, case, monkeypatch):
    vg = astra.create_vol_geom(24, 30, 20)
    v = _vec('cone_vec', 12, 1.0, 1.0)
    if case == "fine":
        v = _vec('cone_vec', 12, 1.0, 0.2)
    elif case == "flipped_rows":
        v[:, 9:12] *= -1
    else:
        v[3, 9] = 0.2
    pg = astra.create_proj_geom('cone_vec', 40, 44, v)
    _check(astra, orc, pg, vg, monkeypatch, gathered=False)


# volumes whose tiles fill the GPU's slots well (16 x 16 blocks and 8 x 8 ones)
FULL = ((256, 256, 128, 60), (192, 192, 192, 60))


def test_default_size(astra, orc):
    """Where the tiles fill the GPU, dense projections are gathered and need no
    scatter."""
    for nx, ny, nz, na in FULL:
        n = nx
        vg = astra.create_vol_geom(ny, nx, nz)
        pg = astra.create_proj_geom('cone', 1.0, 1.0, nz + nz // 4, n + n // 4, np.linspace(0, 2 * np.pi, na, endpoint=False),
                                    4.0 * n, n)
        pr = astra.Projector3D(pg, vg, {'ProjectionKernel': 'matched_bp'})
        x = torch.randn(pr.vol_shape, device='cuda')
        y = torch.rand(pr.proj_shape, device='cuda')
        ax, aty = torch.zeros_like(y), torch.zeros_like(x)
        pr.fp(x, ax)
        _scatters()
        pr.bp(y, aty)
        assert _scatters() == 0
        lhs, rhs = float((ax.double() * y.double()).sum()), float((x.double() * aty.double()).sum())
        assert abs(lhs - rhs) < 1e-6 * float(ax.double().norm() * y.double().norm())


@pytest.mark.parametrize("value", [float('nan'), float('inf'), -float('inf')])
@pytest.mark.parametrize("dtype", ["float32", "float16"])
@pytest.mark.parametrize("pv", [0.45, 0.95, 1.3])
def test_non_finite_values(astra, orc, pv, dtype, value, monkeypatch):
    """A dead pixel reaches the voxels that its ray meets and no others: in
    the detector's first and last rows (rows past them are read with the
    weight zero, for voxels below and above the detector's coverage) and inside
    it.  (Weights below 1e-4 of a ray's largest one may round to nothing.)"""
    vg = astra.create_vol_geom(24, 30, 70)
    pg = astra.create_proj_geom('cone_vec', 41, 53, _vec('cone_vec', 9, 1.0, pv, shift=(1.3, -0.7)))
    pr = astra.Projector3D(pg, vg, {'ProjectionKernel': 'matched_bp'})
    rng = np.random.default_rng(4)
    proj = rng.standard_normal(pr.proj_shape).astype(np.float32)
    dead = np.zeros(pr.proj_shape, dtype=np.float32)
    for pos in ((0, 2, 25), (40, 2, 31), (17, 5, 20), (0, 7, 3)):
        dead[pos] = 1.0
    back = lambda p: orc.fp3d_transpose(pr.geom.kind, pr.geom.views_array(), p, pr.vol_shape, pr.geom.vol_scale)
    weight = back(dead)
    met, missed = weight > 1e-4 * weight.max(), weight == 0
    assert met.any() and missed.any()
    tp = torch.from_numpy(np.where(dead > 0, np.float32(value), proj)).cuda().to(getattr(torch, dtype))
    finite = np.where(dead > 0, 0.0, tp.float().cpu().numpy()).astype(np.float32)
    ref = back(finite)
    for path, name in (("B2T_MATCHED_PATH", "gather"), ("B2T_MATCHED_PLAIN", "1")):
        monkeypatch.setenv(path, name)
        _scatters()
        out = torch.zeros(pr.vol_shape, device='cuda', dtype=tp.dtype)
        pr.bp(tp, out)
        monkeypatch.delenv(path)
        assert (_scatters() == 0) == (name == "gather")
        got = out.float().cpu().numpy()
        assert not np.isfinite(got[met]).any(), path
        assert np.isfinite(got[missed]).all(), path
        assert rel_l2(got[missed], ref[missed]) < {"float32": 1e-5, "float16": 1e-3}[dtype]


def _default(astra, vol, na, du, dv, px=1.0, so=4.0, od=1.0):
    nx, ny, nz = vol
    pg = astra.create_proj_geom('cone', px, px, dv, du, np.linspace(0, 2 * np.pi, na, endpoint=False), so * nx, od * nx)
    return astra.Projector3D(pg, astra.create_vol_geom(ny, nx, nz), {'ProjectionKernel': 'matched_bp'})


@pytest.mark.parametrize("vol,na,du,dv,px", [
    ((64, 64, 64), 1200, 80, 80, 1.0),      # blocks that do not fill the slots
    ((192, 192, 130), 100, 240, 170, 1.0),  # tiles past the volume's last slice
    ((256, 256, 128), 60, 320, 80, 1.0),    # rows for part of the volume
    ((256, 256, 128), 60, 100, 60, 3.0),    # columns and rows far apart
    ((192, 192, 192), 20, 240, 240, 1.0),   # little work
])
def test_default_scatters_where_the_gather_is_slower(astra, vol, na, du, dv, px):
    pr = _default(astra, vol, na, du, dv, px)
    y, x = torch.rand(pr.proj_shape, device='cuda'), torch.zeros(pr.vol_shape, device='cuda')
    _scatters()
    pr.bp(y, x)
    assert _scatters() > 0


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("keep", [0.0, 0.5, 0.87, 0.93, 1.0])
def test_choice_by_the_share_of_values(astra, keep, mode, dtype, monkeypatch):
    """Projections with a value on nine rays in ten or more are gathered, others
    scattered, with the values of the other choice."""
    pr = _default(astra, FULL[1][:3], FULL[1][3], 240, 240)
    t = getattr(torch, dtype)
    gen = torch.Generator('cuda').manual_seed(int(100 * keep))
    y = torch.rand(pr.proj_shape, device='cuda', generator=gen) + 0.5
    y = (y * (torch.rand(pr.proj_shape, device='cuda', generator=gen) < keep)).to(t)
    base = torch.rand(pr.vol_shape, device='cuda', generator=gen).to(t)
    out = {}
    for path in (None, "gather", "scatter"):
        if path:
            monkeypatch.setenv("B2T_MATCHED_PATH", path)
        out[path] = base.clone()
        _scatters()
        pr.bp(y, out[path], mode=mode)
        n = _scatters()
        assert (n == 0) == (keep > 0.9 if path is None else path == "gather")
    monkeypatch.delenv("B2T_MATCHED_PATH")
    a, b, c = (out[k].double() for k in (None, "gather", "scatter"))
    # the scatter's order differs from call to call by 1e-7, which one value in two
    # thousand (FP16) rounds apart, by 2^-10
    again = {"float32": 1e-6, "float16": 1e-4, "bfloat16": 1e-3}[dtype]
    assert torch.equal(a, b) if keep > 0.9 else float((a - c).norm()) <= again * float(c.norm())
    # FP32 sums in another order, and one rounding of the output
    tol = {"float32": 1e-5, "float16": 1e-3, "bfloat16": 8e-3}[dtype]
    assert float((b - c).norm()) <= tol * float(c.norm())


def test_choice_is_made_at_each_replay(astra):
    """A captured call holds both ways and chooses by the projections of the replay."""
    pr = _default(astra, FULL[1][:3], FULL[1][3], 240, 240)
    y, x = torch.rand(pr.proj_shape, device='cuda') + 0.5, torch.zeros(pr.vol_shape, device='cuda')
    pr.bp(y, x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pr.bp(y, x)
    for keep in (1.0, 0.3, 1.0):
        y.copy_((torch.rand_like(y) + 0.5) * (torch.rand_like(y) < keep))
        want = pr.bp(y, torch.zeros_like(x))
        x.fill_(-3.0)
        _scatters()
        graph.replay()
        torch.cuda.synchronize()
        assert (_scatters() == 0) == (keep == 1.0)
        assert float((x - want).norm()) <= 1e-6 * float(want.norm())
