"""Host-pointer calls whose plan has one atlas group: uploads in plane ranges beside the fusion, with the
device call's result bit for bit; and groups of small stacks uploaded several at a time."""
import time

import numpy as np
import pytest
import torch

import pseudoctimaging_b200 as pct

pytestmark = pytest.mark.gpu
DIV = 337.5


def volumes(nx, ny, nz, num, seed, pinned):
    g = torch.Generator().manual_seed(seed)
    base = torch.rand(nz, nx, ny, generator=g) * 300
    v = [base + torch.randn(nz, nx, ny, generator=g) * 3,
         base + torch.randn(num, nz, nx, ny, generator=g) * 3, torch.rand(num, nz, nx, ny, generator=g) * 2000 - 1000]
    return [t.pin_memory() if pinned else t for t in v]


def device(h, v, nh, out):
    num, nz, nx, ny = v[1].shape
    h.synthesize_device(*(t.data_ptr() for t in v), out.data_ptr(), nx, ny, nz, num, nh, DIV,
                        pct.EXEC_B200_FP32)


# one group: aligned and repacked rows, few z-tiles, one range that reads almost all planes; then small
# groups, whole windows and split ones
@pytest.mark.parametrize("nx,ny,nz,num,nh,one", [
    (160, 160, 80, 3, 5, True), (170, 171, 80, 3, 5, True), (188, 149, 46, 5, 7, True),
    (71, 215, 34, 6, 3, True), (150, 160, 33, 4, 3, True), (140, 128, 130, 1, 3, True), (43, 47, 34, 8, 3, False),
    (49, 39, 32, 8, 3, False), (64, 64, 32, 4, 7, False), (38, 103, 41, 7, 3, False),
    (60, 41, 40, 13, 3, False)])
@pytest.mark.parametrize("pinned", [True, False])
def test_parts_equal_one_launch(nx, ny, nz, num, nh, one, pinned):
    assert (pct.query_plan(nx, ny, nz, num, nh)["groups"] == 1) == one
    with pct.Handle(0) as h:
        for seed in (1, 2):
            v = volumes(nx, ny, nz, num, seed, pinned)
            out = torch.zeros(nz, nx, ny, device="cuda")
            device(h, [t.cuda() for t in v], nh, out)
            h.device_status()
            ref = out.cpu().numpy()
            a = [t.numpy() for t in v]
            for _ in range(2):
                np.testing.assert_array_equal(h.synthesize(*a, nh, DIV, pct.EXEC_B200_FP32), ref)
            lab = torch.from_numpy(pct.normalize_labels(a[2])).cuda()
            out.zero_()
            device(h, [v[0].cuda(), v[1].cuda(), lab], nh, out)
            got = h.run_pipeline(*a, nh, 2.5, 1.0, pct.EXEC_B200_FP32, regularize=False)
            np.testing.assert_array_equal(got, out.cpu().numpy())
            full = h.run_pipeline(*a, nh, 2.5, 1.0, pct.EXEC_B200_FP32, regularize=True)
            h.regularize_device(out.data_ptr(), nx, ny, nz, nh)
            h.finalize_hu_device(out.data_ptr(), out.numel())
            np.testing.assert_array_equal(full, out.cpu().numpy())


def test_one_group_overlaps_its_uploads():
    """222x222x112, 2 atlases, NH 7, pinned: 3.7 ms; 4.4 with copies of whole stacks around the device call
    and no repack of their own, 5.2 in one piece with it."""
    nx, ny, nz, num, nh = 222, 222, 112, 2, 7
    assert pct.query_plan(nx, ny, nz, num, nh)["groups"] == 1
    v = volumes(nx, ny, nz, num, 3, True)
    a = [t.numpy() for t in v]
    d = [torch.empty_like(t, device="cuda") for t in v]
    out, back = torch.zeros(nz, nx, ny, device="cuda"), torch.zeros(nz, nx, ny).pin_memory()

    def apart(h):
        for x, y in zip(d, v):
            x.copy_(y, non_blocking=True)
        device(h, d, nh, out)
        back.copy_(out, non_blocking=True)
        torch.cuda.synchronize()

    def ms(f):
        times = []
        for _ in range(12):
            t = time.perf_counter()
            f()
            times.append(1e3 * (time.perf_counter() - t))
        return sorted(times)[4]

    with pct.Handle(0) as h:
        whole, parts = ms(lambda: apart(h)), ms(lambda: h.synthesize(*a, nh, DIV, pct.EXEC_B200_FP32))
    assert parts < 0.95 * whole, (parts, whole)
