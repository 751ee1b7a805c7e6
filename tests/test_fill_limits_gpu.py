"""The NaN fill where a median is itself NaN (both infinities in the middle), and where nothing can be
filled: voxels, counts and time, against the rule in sweep order on the CPU; and the memory that its
allocation-free form holds."""
import subprocess
import sys

import numpy as np
import pytest
import torch

import pseudoctimaging_b200 as pct
from conftest import REPO

pytestmark = pytest.mark.gpu


def fill_rule(vol, nh):
    """A NaN voxel takes the median of its non-NaN neighbours, once, if none of its earlier interior
    neighbours is NaN by then (a voxel whose median is NaN counts as filled and stays NaN)."""
    v = vol.copy()
    nz, nx, ny = v.shape
    lo = (nh - 1) // 2 + 1
    earlier = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)][:13]
    inside = lambda z, x, y: lo <= z < nz - lo and lo <= x < nx - lo and lo <= y < ny - lo
    fills = 0
    for z, x, y in np.argwhere(np.isnan(v)):
        if not inside(z, x, y) or any(inside(z + a, x + b, y + c) and np.isnan(v[z + a, x + b, y + c])
                                      for a, b, c in earlier):
            continue
        n = v[z - 1:z + 2, x - 1:x + 2, y - 1:y + 2].ravel()
        n = np.sort(n[~np.isnan(n)])
        if n.size == 0:
            continue
        with np.errstate(invalid="ignore"):
            v[z, x, y] = n[n.size // 2] if n.size % 2 else np.float32(
                (np.float64(n[n.size // 2 - 1]) + np.float64(n[n.size // 2])) / 2)
        fills += 1
    return v, fills


def run(vol, nh):
    nz, nx, ny = vol.shape
    d = torch.from_numpy(vol).cuda()
    with pct.Handle(0) as h:
        fills = h.regularize_device(d.data_ptr(), nx, ny, nz, nh)
    return d.cpu().numpy(), fills


def check(vol, nh):
    got, fills = run(vol, nh)
    ref, want = fill_rule(vol, nh)
    np.testing.assert_array_equal(got, ref)  # (NaN equal to NaN)
    assert fills == want


def test_first_median_is_nan_and_holds_the_rest():
    vol = np.full((11, 11, 11), np.inf, np.float32)
    vol[:, :, :4] = -np.inf
    box = vol[3:6, 3:6, 3:6].reshape(-1)
    box[:] = np.inf
    box[:9] = -np.inf  # 18 border neighbours of the first voxel left: nine of each sign
    vol[3:6, 3:6, 3:6] = box.reshape(3, 3, 3)
    vol[5, 5, 3] = np.nan
    vol[4:7, 4:7, 4:7] = np.nan
    ref, fills = fill_rule(vol, 7)
    assert fills == 1 and np.isnan(ref[4:7, 4:7, 4:7]).all()
    check(vol, 7)


# chain: NaN voxels in one row, each waiting for the one before it; boxes: single NaN voxels with
# 13 neighbours at either infinity
@pytest.mark.parametrize("chain,boxes", [(1096, 1500), (310, 1500), (40, 3)])
def test_nan_medians_beside_a_chain(chain, boxes):
    vol = np.random.default_rng(chain).normal(50, 20, (20, 40, 1100)).astype(np.float32)
    vol[2, 2, 2:2 + chain] = np.nan
    box = np.full(27, -np.inf, np.float32)
    box[13], box[14:] = np.nan, np.inf
    places = [(z, x, y) for z in (6, 9, 12, 15) for x in range(5, 36, 3) for y in range(4, 1090, 3)]
    for z, x, y in places[:boxes]:
        vol[z - 1:z + 2, x - 1:x + 2, y - 1:y + 2] = box.reshape(3, 3, 3)
    ref, fills = fill_rule(vol, 3)
    assert fills == chain + boxes and not np.isnan(ref[2, 2]).any()
    check(vol, 3)


@pytest.mark.parametrize("shape,nh", [((112, 222, 222), 7), ((40, 90, 100), 3)])
def test_what_nothing_can_fill_ends_soon(shape, nh):
    """All NaN: each launch only looks. Measured 0.77 ms for the larger volume, 0.88 with a launch
    per round; 76 ms when every look of a launch was taken."""
    vol = torch.full(shape, float("nan"), device="cuda")
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    with pct.Handle(0) as h:
        for _ in range(4):
            a.record()
            assert h.regularize_device(vol.data_ptr(), shape[1], shape[2], shape[0], nh) == 0
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
    assert bool(vol.isnan().all())
    assert min(times[1:]) < 8.0, times


NOALLOC = """
import ctypes
import torch
import pseudoctimaging_b200 as pct
n = 1 << 23
v = torch.zeros(n, device="cuda")
v[n // 2 + 64 * 128 + 64] = float("nan")
with pct.Handle(0) as h:  # (the fill's own code is loaded)
    h.regularize_device(torch.zeros(16 ** 3, device="cuda").data_ptr(), 16, 16, 16, 7)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
f = ctypes.c_int64(-1)
st = pct.lib.pct_regularize_device_noalloc(v.data_ptr(), 128, 128, 512, 7, ctypes.byref(f), None)
used = (free - torch.cuda.mem_get_info()[0]) / 2 ** 20
print(st, f.value, int(v.isnan().sum()), used)
"""


def test_noalloc_form_holds_one_list():
    """The largest volume it takes, in a process of its own: 32 MiB of index list."""
    out = subprocess.run([sys.executable, "-c", NOALLOC], cwd=REPO, check=True, capture_output=True,
                         text=True, timeout=120).stdout.split()
    assert out[:3] == ["0", "1", "0"]
    assert 30 <= float(out[3]) <= 40, out
