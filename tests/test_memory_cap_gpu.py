"""Optional scratch (partial sums, stacks repacked for a faster path) under a memory cap: it gives way to
what later calls need, whatever order the calls come in and whatever handles were closed before."""
import numpy as np
import pytest
import torch

import pseudoctimaging_b200 as pct

pytestmark = pytest.mark.gpu
DIV = 337.5
OUT_OF_MEMORY = -3


def volumes(nx, ny, nz, num, seed=1):
    g = torch.Generator().manual_seed(seed)
    base = torch.rand(nz, nx, ny, generator=g) * 300
    return [base + torch.randn(nz, nx, ny, generator=g) * 3,
            base + torch.randn(num, nz, nx, ny, generator=g) * 3, torch.rand(num, nz, nx, ny, generator=g) * 255]


def fill(h):
    """The NaN fill of a 64x72x48 volume: 0.88 MB of scratch."""
    v = torch.rand(48, 64, 72, device="cuda")
    v[20, 30, 30] = float("nan")
    assert h.regularize_device(v.data_ptr(), 64, 72, 48, 7) == 1


def device(nx, ny, nz, num, nh, choice, k=0):
    def go(h):
        d = [t.contiguous().cuda() for t in volumes(nx, ny, nz, num)]
        out = torch.zeros_like(d[0])
        if k:
            h.set_learned_prior(k)
        h.synthesize_device(*(t.data_ptr() for t in d), out.data_ptr(), nx, ny, nz, num, nh, DIV, choice)
        h.device_status()
        return out.cpu().numpy()
    return go


def host(nx, ny, nz, num, nh):
    a = [t.numpy() for t in volumes(nx, ny, nz, num)]
    return lambda h: h.synthesize(*a, nh, DIV, pct.EXEC_B200_FP32)


class Batch:
    """Captures a batch of one subject, runs it once and leaves it alive on its handle."""

    def __init__(self, nx, ny, nz, num, nh):
        self.shape, self.nh, self.alive = (nx, ny, nz, num), nh, []

    def __call__(self, h):
        d = [t.contiguous().cuda() for t in volumes(*self.shape)]
        out = torch.zeros_like(d[0])
        nx, ny, nz, num = self.shape
        b = h.batch_graph([dict(img=d[0].data_ptr(), atlas=d[1].data_ptr(), atlas_label=d[2].data_ptr(),
                                out=out.data_ptr(), nx=nx, ny=ny, nz=nz, num_atlas=num, nh=self.nh,
                                div=DIV)])
        self.alive.append((b, d))
        b.launch()
        b.status()
        return out.cpu().numpy()

    def close(self):
        for b, _ in self.alive:
            b.close()
        self.alive.clear()


def fits(calls, cap):
    """The calls' results on a handle with this cap, None if one does not fit."""
    with pct.Handle(0) as h:
        h.set_memory_limit(cap)
        try:
            return [c(h) for c in calls]
        except pct.PctError as e:
            assert e.status == OUT_OF_MEMORY
            return None
        finally:
            for c in calls:
                if isinstance(c, Batch):
                    c.close()  # (before its handle)


def same(a, b):
    """Equal up to the order of FP32 sums, each within 1e-4 of the exact value as elsewhere."""
    if a is not None:
        np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
        np.testing.assert_allclose(a, b, rtol=2e-4, equal_nan=True)


@pytest.mark.parametrize("call", [
    device(64, 64, 32, 1, 7, pct.EXEC_B200_FP32), device(40, 43, 26, 2, 9, pct.EXEC_B200_FP32),
    device(33, 45, 24, 2, 11, pct.EXEC_LEARNED, 33), host(40, 44, 30, 2, 5), host(40, 43, 30, 3, 5),
    Batch(48, 44, 40, 4, 7)], ids=["split", "split-repack", "prior-repack", "host", "host-repack", "batch"])
def test_what_fits_in_one_order_fits_in_the_other(call):
    with pct.Handle(0) as h:
        ref = call(h)
        if isinstance(call, Batch):
            call.close()
    cap = 900_000
    while fits([fill, call], cap) is None:
        cap += cap // 16
    for limit in (cap, cap + cap // 4, 2 * cap, 4 * cap):
        for calls in ([call, fill], [call, fill, call, fill]):
            outs = fits(calls, limit)
            assert outs is not None, f"out of memory at {limit} bytes where {cap} do in the other order"
            for o in outs:
                same(o, ref)


def test_larger_calls_after_smaller_ones():
    """A 222x222x112 volume and one atlas: 133 MB for the three calls in any order."""
    d = [t.numpy() for t in volumes(222, 222, 112, 1)]
    v = torch.rand(112, 222, 222, device="cuda")
    with pct.Handle(0) as h:
        ref = h.synthesize(*d, 3, DIV, pct.EXEC_B200_FP32)
    with pct.Handle(0) as h:
        h.set_memory_limit(150_000_000)
        device(64, 64, 32, 1, 7, pct.EXEC_B200_FP32)(h)
        device(222, 222, 112, 1, 11, pct.EXEC_B200_FP32)(h)
        h.regularize_device(v.data_ptr(), 222, 222, 112, 11)
        same(h.synthesize(*d, 3, DIV, pct.EXEC_B200_FP32), ref)
        h.regularize_device(v.data_ptr(), 222, 222, 112, 11)


def test_a_closed_handle_takes_no_room_from_a_capped_one():
    """Partial sums that a closed handle left behind are taken over only within the cap."""
    call = host(40, 44, 30, 2, 5)
    cap = 100_000
    while fits([call], cap) is None:
        cap += cap // 16
    limit = cap
    with pct.Handle(0):
        while limit < 8 * cap:
            for nz in (16, 24, 32, 48):  # blocks of several sizes are left behind
                with pct.Handle(0) as h:
                    device(48, 48, nz, 1, 7, pct.EXEC_B200_FP32)(h)
            assert fits([call], limit) is not None, f"out of memory at {limit} bytes; {cap} are enough"
            limit += limit // 8
