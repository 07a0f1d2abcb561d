"""The row split of the tensor-core Ram-Lak filter and the padding of
projections at the edges of their tiles: rows around multiples of 8 and of the
256-column chunks, a last CTA of one to four rows, fewer views than rows of a
CTA, view counts around the 8 and 32 views of a padding thread and block."""
import ctypes
import importlib

import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# FP32 sums of a few hundred terms: about 1e-6; 1e-5 as in the other filter tests
@pytest.mark.parametrize("nu", [127, 128, 129, 255, 256, 257, 263, 264, 265, 513, 832])
@pytest.mark.parametrize("nrows", [128, 129, 130, 131])
def test_rows(astra, orc, nu, nrows):
    lib = importlib.import_module("astra-toolbox_b200._lib").load()
    P = importlib.import_module("astra-toolbox_b200.projector")
    x = np.random.default_rng(nu).random((nrows, nu + 3), dtype=np.float32)
    buf = torch.from_numpy(x).cuda()
    cfg = P.FilterSpec('ram-lak').c()
    st = lib.b2t_filter_rows(buf.data_ptr(), nrows, nu, nu + 3, ctypes.byref(cfg),
                             torch.cuda.current_stream().cuda_stream)
    assert st == 0, lib.b2t_last_error()
    want = x[:, :nu].astype(np.float64)
    want = np.ascontiguousarray(want)
    orc.ramp_filter_rows(want)
    got = buf.cpu().numpy()
    assert rel_l2(got[:, :nu], want) < 1e-5
    assert np.array_equal(got[:, nu:], x[:, nu:])


# FP32: positions of up to 133 texels are off by about 133 x 2^-23 = 1.6e-5
# texels, and neighbouring texels of filtered white noise differ by about
# sqrt(2) of their norm, so 2.2e-5 where no average over views hides it
@pytest.mark.parametrize("na", [1, 2, 3, 5])
@pytest.mark.parametrize("dtype,tol", [("float32", 3e-5), ("float16", 2e-3), ("bfloat16", 1.5e-2)])
def test_few_views_and_fdk_border(astra, orc, na, dtype, tol):
    P = importlib.import_module("astra-toolbox_b200.projector")
    ang = np.linspace(0, 2 * np.pi, na, endpoint=False).astype(np.float32)
    vg = astra.create_vol_geom(40, 36, 30)
    pg = astra.create_proj_geom('cone', 0.4, 1.0, 131, 133, ang, 200.0, 100.0)
    pr = P.Projector3D(pg, vg)
    proj = torch.from_numpy(np.random.default_rng(na).random(pr.proj_shape, dtype=np.float32)).cuda().to(
        getattr(torch, dtype))
    rec = torch.zeros(pr.vol_shape, device='cuda', dtype=proj.dtype)
    # the scratch that the call gets back held other values
    P.fdk(pr, torch.full_like(proj, 3.0e4), torch.zeros_like(rec))
    P.fdk(pr, proj, rec)
    ref = orc.fdk(pr.geom.views_array(), proj.float().cpu().numpy(), pr.vol_shape, pr.geom.vol_scale)
    assert rel_l2(rec.float().cpu().numpy(), ref) < tol


@pytest.mark.parametrize("na", [1, 7, 8, 9, 31, 32, 33])
@pytest.mark.parametrize("dtype,tol", [("float32", 1e-5), ("float16", 2e-3), ("bfloat16", 1.5e-2)])
def test_padding(astra, orc, na, dtype, tol):
    ang = np.linspace(0, 2 * np.pi, na, endpoint=False).astype(np.float32)
    vg = astra.create_vol_geom(20, 24, 18)
    for nu in (27, 28, 29, 61):
        pg = astra.create_proj_geom('cone', 1.1, 0.8, 23, nu, ang, 90.0, 40.0)
        pr = astra.Projector3D(pg, vg)
        proj = torch.from_numpy(np.random.default_rng(nu).random(pr.proj_shape, dtype=np.float32)).cuda().to(
            getattr(torch, dtype))
        rec = torch.zeros(pr.vol_shape, device='cuda', dtype=proj.dtype)
        pr.bp(proj, rec)
        ref = orc.bp3d(pr.geom.kind, pr.geom.views_array(), proj.float().cpu().numpy(), pr.vol_shape,
                       pr.geom.vol_scale)
        assert rel_l2(rec.float().cpu().numpy(), ref) < tol, nu
