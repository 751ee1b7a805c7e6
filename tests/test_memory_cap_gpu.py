"""Optional scratch under a memory cap: what a call needs fits whatever handles were closed before."""
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


def fits(calls, cap):
    """The calls' results on a handle with this cap, None if one does not fit."""
    with pct.Handle(0) as h:
        h.set_memory_limit(cap)
        try:
            return [c(h) for c in calls]
        except pct.PctError as e:
            assert e.status == OUT_OF_MEMORY
            return None


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
