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
def test_16_bit_storage_rounds_the_fp32_projection(astra, dtype, kind):
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
