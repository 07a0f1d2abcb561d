"""The 2D projectors on lines of texel pairs (csrc/lines2d.cu) against the
direct bodies, bit for bit: both evaluate the same positions, samples and
partial sums.  A failed scratch allocation sends a forward projection to the
direct kernels; the batched backprojection runs the direct body (one chunk of
1024 views at most is summed alike)."""
import importlib

import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _vec(kind, n, seed):
    """Uneven orbits whose detectors are offset, tilted and of varying pitch."""
    rng = np.random.default_rng(seed)
    out = np.zeros((n, 6))
    for i in range(n):
        t = 2 * np.pi * i / n + rng.normal(0, 0.05)
        w = rng.uniform(0.7, 1.4)
        c, s = np.cos(t), np.sin(t)
        tilt = t + rng.normal(0, 0.05)
        u = [w * np.cos(tilt), w * np.sin(tilt)]
        if kind == 'parallel_vec':
            out[i] = [-s, c, rng.normal(0, 3), rng.normal(0, 3), *u]
        else:
            out[i] = [90 * s, -90 * c, -45 * s, 45 * c, *u]
    return out


# (kind, rows, cols, views, dets): one pixel, edges of the 32-texel and
# 64-detector tiles and one past them, a detector narrower than the image
# (clamped backprojection) and wider, launches over 1024 views, sizes of every
# split of the slices (warps below 1200, below 2400, above) and of the views
SHAPES = [
    ('parallel', 1, 1, 1, 1), ('parallel', 3, 2, 5, 7), ('parallel', 32, 32, 9, 64), ('parallel', 33, 31, 17, 65),
    ('parallel', 128, 128, 180, 192), ('parallel', 90, 250, 500, 260), ('parallel', 230, 230, 1030, 129),
    ('parallel', 300, 710, 40, 500), ('parallel', 60, 64, 200, 20), ('parallel_vec', 65, 97, 61, 200),
    ('fanflat', 64, 64, 40, 96), ('fanflat', 31, 77, 33, 63), ('fanflat', 257, 129, 700, 400),
    ('fanflat', 900, 850, 30, 1301), ('fanflat', 80, 80, 1100, 25), ('fanflat_vec', 50, 61, 77, 150),
    # detectors so fine that a tile's footprint exceeds the staged window
    ('parallel_fine', 40, 44, 50, 900), ('fanflat_fine', 40, 44, 50, 900),
    # small images of more than 64 views, whose projections go through lines as well
    ('parallel', 1, 1, 70, 1), ('parallel', 3, 2, 65, 7), ('parallel', 32, 32, 69, 64), ('parallel', 33, 31, 77, 65),
    ('fanflat', 1, 1, 66, 3), ('fanflat', 64, 64, 65, 96), ('parallel_fine', 40, 44, 70, 900), ('fanflat_fine', 40, 44, 70, 900),
]


def _problem(astra, kind, rows, cols, views, dets):
    ang = np.linspace(0, 2 * np.pi, views, endpoint=False).astype(np.float32)
    vg = astra.create_vol_geom(rows, cols)
    n = max(rows, cols)
    if kind == 'parallel_fine':
        return vg, astra.create_proj_geom('parallel', 0.07, dets, ang)
    if kind == 'fanflat_fine':
        return vg, astra.create_proj_geom('fanflat', 0.1, dets, ang, 1.5 * n, 0.7 * n)
    if kind == 'parallel':
        return vg, astra.create_proj_geom('parallel', 1.0, dets, ang)
    if kind == 'fanflat':
        return vg, astra.create_proj_geom('fanflat', 1.3, dets, ang, 1.5 * n, 0.7 * n)
    return vg, astra.create_proj_geom(kind, dets, _vec(kind, views, rows))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("rays", [1, 2])
def test_lines_equal_direct(astra, orc, shape, rays):
    lib = importlib.import_module("astra-toolbox_b200._lib").load()
    vg, pg = _problem(astra, *shape)
    pr = astra.Projector2D(pg, vg, {'DetectorSuperSampling': rays})
    rng = np.random.default_rng(5)
    vol, sino = rng.random(pr.vol_shape, dtype=np.float32), rng.random(pr.proj_shape, dtype=np.float32)
    tv, ts = torch.from_numpy(vol).cuda(), torch.from_numpy(sino).cuda()

    def both(call, out):
        got = []
        for fail in (0, 1):
            t = torch.full(out, 0.25, device='cuda')
            lib.b2t_debug_fail_alloc(fail, None)
            try:
                call(t)
            finally:
                lib.b2t_debug_fail_alloc(0, None)
            got.append(t)
        assert torch.equal(got[0], got[1])
        return got[0]

    fp = both(lambda t: pr.fp(tv, t), pr.proj_shape)
    both(lambda t: pr.fp(tv, t, mode=0), pr.proj_shape)
    fan = pr.geom.kind == 4
    if shape[1] * shape[2] * shape[3] < 2_000_000:
        f = orc.fan_fp if fan else orc.par_fp
        ref = f(pr.geom.views_array(), vol, shape[4], pr.geom.output_scale, rays=rays)
        assert np.linalg.norm(fp.cpu().numpy() - ref) <= 1e-5 * np.linalg.norm(ref)
    if rays > 1:
        return
    bp = torch.full(pr.vol_shape, 0.25, device='cuda')
    pr.bp(ts, bp)
    B = astra.Batch2D([(pg, vg)])
    direct = B.vol_views(B.bp(B.pack_sinos([ts])))[0]
    if shape[3] <= 1024:
        assert torch.equal(bp, direct)
    else:
        assert float((bp - direct).norm()) <= 1e-6 * float(direct.norm())
    B.close()
    add = torch.full(pr.vol_shape, 0.25, device='cuda')
    pr.bp(ts, add, mode=0)
    assert torch.allclose(add, bp + 0.25, rtol=1e-6, atol=0)
    if fan:
        w = torch.zeros(pr.vol_shape, device='cuda')
        pr.bp(ts, w, fbp_weight=True)
        if shape[1] * shape[2] * shape[3] < 2_000_000:
            ref = orc.fan_bp(pr.geom.views_array(), sino, pr.vol_shape, pr.geom.output_scale, fbp=True)
            assert rel_l2(w.cpu().numpy(), ref) < 1e-5
    if shape[1] * shape[2] * shape[3] < 2_000_000:
        b = orc.fan_bp if fan else orc.par_bp
        ref = b(pr.geom.views_array(), sino, pr.vol_shape, pr.geom.output_scale)
        assert rel_l2(bp.cpu().numpy(), ref) < 1e-5


def test_lines_take_pitched_rows_and_odd_addresses(astra):
    """Row pitches above the row length and 4-byte-aligned bases, through the
    C entry points."""
    import ctypes
    L = importlib.import_module("astra-toolbox_b200._lib")
    vg, pg = _problem(astra, 'fanflat', 37, 53, 29, 71)
    pr = astra.Projector2D(pg, vg)
    vol = torch.rand(pr.vol_shape, device='cuda')
    sino = torch.rand(pr.proj_shape, device='cuda')
    want_fp, want_bp = torch.zeros_like(sino), torch.zeros_like(vol)
    pr.fp(vol, want_fp)
    pr.bp(sino, want_bp)

    def pitched(t):
        buf = torch.full((t.shape[0] * (t.shape[1] + 6) + 1,), -7.0, device='cuda')
        v = buf[1:].view(t.shape[0], -1)
        v[:, :t.shape[1]] = t
        return buf, v

    bv, v = pitched(vol)
    bs, s = pitched(sino)
    L.call("b2t_fp2d", ctypes.byref(pr.geom.c), 1, v.data_ptr(), 59, s.data_ptr(), 77, 1, None)
    torch.cuda.synchronize()
    assert torch.equal(s[:, :71], want_fp) and bool((s[:, 71:] == -7.0).all())
    _, s = pitched(sino)
    L.call("b2t_bp2d", ctypes.byref(pr.geom.c), 1, 0, s.data_ptr(), 77, v.data_ptr(), 59, 1, None)
    torch.cuda.synchronize()
    assert torch.equal(v[:, :53], want_bp) and bool((v[:, 53:] == -7.0).all())
