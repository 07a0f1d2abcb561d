"""The slab forward projector over detector heights at the edges of its row
blocks, slice counts at the edges of its stages and volumes thinner and
thicker than its boxes, against the cell kernels; 16-bit storage is the FP32
projection of the same values, rounded once."""
import ctypes
import importlib

import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _stats(L):
    out = (ctypes.c_uint64 * 4)()
    assert L.load().b2t_fp_path_stats(out) == 0
    return list(out)


@pytest.mark.parametrize("rows", [1, 32, 33, 129, 160, 161, 192, 330])
@pytest.mark.parametrize("vol", [(1, 1, 1), (2, 3, 7), (33, 32, 5), (31, 64, 40), (40, 34, 230)])
@pytest.mark.parametrize("kind", ["cone", "parallel3d"])
def test_row_blocks_and_stages(astra, rows, vol, kind, monkeypatch):
    L = importlib.import_module("astra-toolbox_b200._lib")
    ny, nx, nz = vol
    ang = np.linspace(0, 2 * np.pi, 17, endpoint=False).astype(np.float32)
    vg = astra.create_vol_geom(ny, nx, nz)
    n = max(ny, nx, 8)
    px = 1.2 * max(nz, 4) / max(rows, 8) + 0.3
    if kind == "cone":
        pg = astra.create_proj_geom('cone', 1.1, px, rows, 49, ang, 2.5 * n, 1.0 * n)
    else:
        pg = astra.create_proj_geom('parallel3d', 0.8, px, rows, 49, ang)
    pr = astra.Projector3D(pg, vg)
    tv = torch.from_numpy(np.random.default_rng(rows).random(pr.vol_shape, dtype=np.float32)).cuda()
    _stats(L)
    a = torch.zeros(pr.proj_shape, device='cuda')
    pr.fp(tv, a)
    assert _stats(L)[3] == 0
    flags = ctypes.c_uint32(1)
    assert L.load().b2t_device_errors(ctypes.byref(flags)) == 0 and flags.value == 0
    monkeypatch.setenv("B2T_FP_PATH", "cells")
    b = torch.zeros(pr.proj_shape, device='cuda')
    pr.fp(tv, b)
    monkeypatch.delenv("B2T_FP_PATH")
    assert float(b.abs().max()) > 0
    assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 2e-6


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("kind", ["cone", "parallel3d"])
def test_16_bit_storage_rounds_the_fp32_projection(astra, dtype, kind, monkeypatch):
    monkeypatch.setenv("B2T_FP_PATH", "slab")  # (so few views are faster from cells)
    L = importlib.import_module("astra-toolbox_b200._lib")
    t = getattr(torch, dtype)
    ang = np.linspace(0, 2 * np.pi, 25, endpoint=False).astype(np.float32)
    vg = astra.create_vol_geom(37, 45, 50)
    if kind == "cone":
        pg = astra.create_proj_geom('cone', 1.1, 1.2, 65, 71, ang, 110.0, 60.0)
    else:
        pg = astra.create_proj_geom('parallel3d', 0.9, 0.9, 65, 71, ang)
    pr = astra.Projector3D(pg, vg)
    tv = torch.from_numpy(np.random.default_rng(3).random(pr.vol_shape, dtype=np.float32)).cuda().to(t)
    _stats(L)
    half = torch.zeros(pr.proj_shape, device='cuda', dtype=t)
    pr.fp(tv, half)
    assert _stats(L)[3] == 0, "the slab kernel takes 16-bit volumes"
    full = torch.zeros(pr.proj_shape, device='cuda')
    pr.fp(tv.float(), full)
    assert torch.equal(half, full.to(t))
    # ADD reads and rounds the stored projections
    base = torch.rand(pr.proj_shape, device='cuda').to(t)
    add = base.clone()
    pr.fp(tv, add, mode=0)
    assert torch.equal(add, (full + base.float()).to(t))


# (views, detector columns, rows, volume, slab): enough CTAs of enough rows; too
# few CTAs, too few rows in each, neighbouring views too far apart for a slice
# buffer, a source so close that the rays of a CTA leave the volume one by one
CHOICES = {
    "many": (430, 110, 90, (64, 64, 70), 1.2, 2.0, True),
    "tall": (220, 130, 125, (90, 90, 100), 1.2, 2.0, True),
    "few_views": (120, 110, 90, (64, 64, 70), 1.2, 2.0, False),
    "few_rows": (430, 110, 60, (64, 64, 40), 1.2, 2.0, False),
    "far_views": (44, 900, 150, (300, 300, 100), 0.6, 2.0, False),
    "near_source": (430, 110, 130, (64, 64, 64), 5.0, 0.75, False),
}


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("case", list(CHOICES))
def test_16_bit_choice_of_kernel(astra, case, dtype, monkeypatch):
    """Which 16-bit scans take the slab, with the other choice's values; FP32
    ones all do."""
    L = importlib.import_module("astra-toolbox_b200._lib")
    views, nu, nv, (ny, nx, nz), px, so, slab = CHOICES[case]
    ang = np.linspace(0, 2 * np.pi, views, endpoint=False).astype(np.float32)
    od = 3.0 if so < 1 else 1.0
    pg = astra.create_proj_geom('cone', px, px, nv, nu, ang, so * nx, od * nx)
    pr = astra.Projector3D(pg, astra.create_vol_geom(ny, nx, nz))
    t = getattr(torch, dtype)
    vol = torch.rand(pr.vol_shape, device='cuda', generator=torch.Generator('cuda').manual_seed(1)).to(t)
    out = {}
    for path in (None, "cells", "slab"):
        if path:
            monkeypatch.setenv("B2T_FP_PATH", path)
        _stats(L)
        out[path] = torch.zeros(pr.proj_shape, device='cuda', dtype=t)
        pr.fp(vol, out[path])
        s = _stats(L)
        assert (s[2] > 0, s[3] > 0) == ((False, True) if path == "cells" or not (path or slab) else (True, False))
    monkeypatch.delenv("B2T_FP_PATH")
    assert torch.equal(out[None], out["slab" if slab else "cells"])
    # one rounding of the output; the cells hold 16-bit differences as well
    tol = {"float16": 1e-3, "bfloat16": 8e-3}[dtype]
    assert rel_l2(out["cells"].float().cpu().numpy(), out["slab"].float().cpu().numpy()) < tol
    full = torch.zeros(pr.proj_shape, device='cuda')
    _stats(L)
    pr.fp(vol.float(), full)
    assert _stats(L)[3] == 0
    assert rel_l2(out["slab"].float().cpu().numpy(), full.cpu().numpy()) < tol


# (volume, views, detector columns, rows, pixel, slab): pixels of 0.8 voxels at the
# volume's middle and of twice their size, few views of them, and views far apart
# that see past the volume and that do not
@pytest.mark.parametrize("vol,views,nu,nv,px,slab", [
    ((150, 150, 150), 200, 200, 180, 1.2, True),
    ((150, 150, 150), 200, 110, 100, 3.0, False),
    ((200, 200, 200), 24, 200, 200, 1.8, False),
    ((200, 200, 200), 32, 250, 250, 1.2, True),
    ((150, 150, 150), 16, 110, 100, 3.0, True),
])
def test_fp32_choice_of_kernel(astra, orc, vol, views, nu, nv, px, slab, monkeypatch):
    """FP32 scans whose slices do not fit the slab's buffers take the cells, with
    the slab's values; a failed allocation of theirs takes the slab."""
    L = importlib.import_module("astra-toolbox_b200._lib")
    nx, ny, nz = vol
    ang = np.linspace(0, 2 * np.pi, views, endpoint=False).astype(np.float32)
    pr = astra.Projector3D(astra.create_proj_geom('cone', px, px, nv, nu, ang, 2.0 * nx, 1.0 * nx),
                           astra.create_vol_geom(ny, nx, nz))
    v = torch.rand(pr.vol_shape, device='cuda', generator=torch.Generator('cuda').manual_seed(2))
    _stats(L)
    a = pr.fp(v, torch.zeros(pr.proj_shape, device='cuda'))
    s = _stats(L)
    assert (s[2] > 0, s[3] > 0) == (slab, not slab)
    monkeypatch.setenv("B2T_FP_PATH", "slab")
    b = pr.fp(v, torch.zeros(pr.proj_shape, device='cuda'))
    monkeypatch.delenv("B2T_FP_PATH")
    assert _stats(L)[3] == 0
    # both round positions and sums in FP32
    assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 2e-6
    if not slab:
        L.load().b2t_debug_fail_alloc(1, None)
        try:
            c = pr.fp(v, torch.zeros(pr.proj_shape, device='cuda'))
        finally:
            L.load().b2t_debug_fail_alloc(0, None)
        assert _stats(L)[3] == 0 and torch.equal(b, c)


@pytest.mark.parametrize("rows", [161, 180, 230, 330, 358])
@pytest.mark.parametrize("nz", [40, 120, 300])
def test_row_blocks_full_and_equal(astra, orc, rows, nz, monkeypatch):
    """Enough CTAs for full blocks of rows and a rest, where these leave more of
    the detector beside the volume's shadow, and equal blocks; short and tall
    volumes, a detector shifted along z."""
    views = 1000
    out = np.zeros((views, 12))
    for i in range(views):
        t = 2 * np.pi * i / views
        u, r = np.array([np.cos(t), np.sin(t), 0.0]), np.array([np.sin(t), -np.cos(t), 0.0])
        out[i] = np.concatenate([r * 60.0, -r * 20.0 + [0.0, 0.0, 13.0], 1.1 * u, [0.0, 0.0, 1.2]])
    pr = astra.Projector3D(astra.create_proj_geom('cone_vec', rows, 33, out), astra.create_vol_geom(20, 18, nz))
    v = torch.rand(pr.vol_shape, device='cuda')
    a = pr.fp(v, torch.zeros(pr.proj_shape, device='cuda'))
    monkeypatch.setenv("B2T_FP_PATH", "cells")
    b = pr.fp(v, torch.zeros(pr.proj_shape, device='cuda'))
    assert float(b.abs().max()) > 0
    assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 2e-6
