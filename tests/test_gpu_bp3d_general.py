"""The TMA backprojector on orbits whose detector coordinates vary along a
voxel column in every respect (tilted detectors, inclined parallel rays),
against the direct-load kernel and the FP64 oracle: columns at the ends of
16- and 32-voxel blocks, small and strong tilts (strong ones leave the tile
and take the per-sample checks), every storage type."""
import ctypes
import importlib

import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _paths():
    """Voxel-column views on the circular path, on others, and of those on the
    packed path, since the last call."""
    lib = importlib.import_module("astra-toolbox_b200._lib").load()
    st, packed = (ctypes.c_uint64 * 4)(), ctypes.c_uint64(0)
    assert lib.b2t_bp_path_stats(st) == 0 and lib.b2t_bp_packed_columns(ctypes.byref(packed)) == 0
    return st[0], st[1], packed.value


def _vectors(kind, n, tilt_deg, seed):
    rng = np.random.default_rng(seed)
    out = np.zeros((n, 12))
    for i in range(n):
        t = 2 * np.pi * i / n + 0.05
        u, v = np.array([np.cos(t), np.sin(t), 0.0]), np.array([0.0, 0.0, 1.0])
        w = np.cross(u, v)
        a, b, c = np.deg2rad(rng.normal(0.0, tilt_deg, 3))
        u2 = u * np.cos(a) + v * np.sin(a) * np.cos(c) + w * np.sin(a) * np.sin(c)
        v2 = v * np.cos(b) + w * np.sin(b)
        off = rng.normal(0, 0.6) * u + rng.normal(0, 0.6) * v
        if kind == 'cone_vec':
            src = np.array([np.sin(t), -np.cos(t), 0.0]) * 130 + v * rng.normal(0, 2)
            out[i] = np.concatenate([src, -src * 0.5 + off, 1.1 * u2, 1.2 * v2])
        else:
            ray = np.array([-np.sin(t), np.cos(t), np.sin(b)])
            out[i] = np.concatenate([ray, off, 1.1 * u2, 1.2 * v2])
    return out


@pytest.mark.parametrize("kind", ["cone_vec", "parallel3d_vec"])
@pytest.mark.parametrize("tilt", [0.1, 4.0, 35.0])
@pytest.mark.parametrize("shape", [(1, 1, 1), (15, 9, 33), (16, 8, 32), (33, 17, 31), (64, 40, 70)])
def test_general_orbits(astra, orc, kind, tilt, shape, monkeypatch):
    nz, ny, nx = shape
    vg = astra.create_vol_geom(ny, nx, nz)
    pg = astra.create_proj_geom(kind, 57, 91, _vectors(kind, 23, tilt, nz))
    rng = np.random.default_rng(nx)
    for opts in [{}] + ([{'ProjectionKernel': '2d_weighting'}] if kind == 'cone_vec' else []):
        pr = astra.Projector3D(pg, vg, opts)
        proj = rng.random(pr.proj_shape, dtype=np.float32)
        tp = torch.from_numpy(proj).cuda()
        got = {}
        for dtype in (torch.float32, torch.float16, torch.bfloat16):
            a = torch.zeros(pr.vol_shape, device='cuda', dtype=dtype)
            _paths()
            pr.bp(tp.to(dtype), a)
            circular, other, packed = _paths()
            assert circular == 0 and other > 0
            if shape == (64, 40, 70):  # (smaller ones cut the columns short of a block)
                share = packed / other
                # (no parallel view of these leaves its tile)
                assert share > 0.99 if tilt == 0.1 or kind == 'parallel3d_vec' else 0.5 < share if tilt == 4.0 else 0.0 < share < 1.0, share
            got[dtype] = a.float().cpu().numpy()
        monkeypatch.setenv("B2T_SIMPLE_BP", "1")
        for dtype, tol in ((torch.float32, 4e-6), (torch.float16, 5e-4), (torch.bfloat16, 4e-3)):
            b = torch.zeros(pr.vol_shape, device='cuda', dtype=dtype)
            pr.bp(tp.to(dtype), b)
            assert rel_l2(got[dtype], b.float().cpu().numpy()) < tol, (dtype, opts)
        monkeypatch.delenv("B2T_SIMPLE_BP")
        kernel = 3 if opts else 0
        ref = orc.bp3d(pr.geom.kind, pr.geom.views_array(), proj, pr.vol_shape, pr.geom.vol_scale, kernel=kernel)
        assert rel_l2(got[torch.float32], ref) < 1e-5, opts
        c = torch.full(pr.vol_shape, 2.0, device='cuda')
        pr.bp(tp, c, mode=0)
        assert rel_l2(c.cpu().numpy() - 2.0, ref) < 1e-5
