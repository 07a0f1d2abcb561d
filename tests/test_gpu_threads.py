"""Calls of the same kernel from several host threads at once.  A kernel's
dynamic shared memory limit belongs to the kernel and not to the call: a call
that set it to what its own launch needs would take it from another thread's
larger launch."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _together(calls, n):
    """n runs of every call, one thread and stream each, begun together; the
    outputs of a last run."""
    gate, errors, outs = threading.Barrier(len(calls), timeout=60), [], [None] * len(calls)

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait()
                for _ in range(n):
                    outs[k] = calls[k]()
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    return outs


def _check(calls, n):
    want = [f().clone() for f in calls]
    for got, ref in zip(_together(calls, n), want):
        assert torch.equal(got, ref)


@pytest.mark.parametrize("n,views", [(64, 5000), (240, 3000), (480, 2000), (600, 2000)])
def test_backprojections_of_different_windows(astra, n, views):
    """Detectors of one pixel and of half a pixel: the same kernel, with
    windows of staged sinogram rows of different widths (sizes of every split
    of the views over warps; several launches a call, so that the threads are
    mostly inside the library)."""
    def call(px):
        ang = np.linspace(0, np.pi, views, endpoint=False)
        pr = astra.Projector2D(astra.create_proj_geom('parallel', px, int(1.5 * n / px), ang),
                               astra.create_vol_geom(n, n))
        sino, vol = torch.rand(pr.proj_shape, device='cuda'), torch.zeros(pr.vol_shape, device='cuda')
        return lambda: pr.bp(sino, vol)

    _check([call(1.0), call(0.5)], 1000 if n < 400 else 300)


@pytest.mark.parametrize("filter_type", ["ram-lak", "hann"])
def test_filters_of_different_rows(astra, filter_type):
    """Few and many rows, short and long: tensor-core tiles of different
    widths, staged rows of different lengths."""
    def call(n, rows):
        ang = np.linspace(0, np.pi, rows, endpoint=False)
        pr = astra.Projector2D(astra.create_proj_geom('parallel', 1.0, n, ang), astra.create_vol_geom(16, 16))
        sino, vol = torch.rand(pr.proj_shape, device='cuda'), torch.zeros(pr.vol_shape, device='cuda')
        return lambda: astra.projector.fbp2d(pr, sino, vol, filter_type=filter_type)

    _check([call(768, 130), call(700, 2600)], 1500 if filter_type == "ram-lak" else 300)
