"""NaN and infinities in the input, the atlases and the labels: the paths that a rule on sizes chooses
(windows split over CTAs, the centre prior on tiles) against the general ones, voxel by voxel."""
import numpy as np
import pytest
import torch

import pseudoctimaging_b200 as pct

pytestmark = pytest.mark.gpu
DIV = 337.5


def volumes(nx, ny, nz, num, seed):
    """Smooth volumes with single NaN, +inf, -inf and FP32 maxima in all three inputs, in the border and
    the interior, and both infinities at one place of the input and an atlas."""
    r = np.random.default_rng(seed)
    base = r.normal(0, 8, (nz, nx, ny)).cumsum(2)
    img = (base + r.normal(0, 2, base.shape)).astype(np.float32)
    mri = (base + r.normal(0, 2, (num,) + base.shape)).astype(np.float32)
    lab = r.uniform(0, 255, mri.shape).astype(np.float32)
    vals = [np.nan, np.inf, -np.inf, 3.4e38, -3.4e38, 0.0]
    for a in (img, mri.reshape(-1, nx, ny), lab.reshape(-1, nx, ny)):
        for k in range(len(vals) * (1 if a is img else num)):
            z, x, y = (int(r.integers(0, n)) for n in a.shape)
            a[z, x, y] = vals[k % len(vals)]
    z, x, y = nz // 2, nx // 2, ny // 2
    img[z, x, y] = mri[0, z, x, y] = np.inf
    img[z - 1, x - 3, y + 2], mri[-1, z - 1, x - 3, y + 2] = -np.inf, np.inf
    return img, mri, lab


def run(h, v, nh, choice):
    num, nz, nx, ny = v[1].shape
    d = [torch.from_numpy(a).cuda() for a in v]
    out = torch.zeros(nz, nx, ny, device="cuda")
    h.synthesize_device(*(t.data_ptr() for t in d), out.data_ptr(), nx, ny, nz, num, nh, DIV, choice)
    h.device_status()
    return out.cpu().numpy()


def same(got, ref):
    """Non-finite voxels the same; the others equal up to the order of FP32 sums (each path is within
    1e-4 of the exact value elsewhere)."""
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_allclose(got, ref, rtol=2e-4, equal_nan=True)
    assert np.isnan(ref).any() and np.isfinite(ref).sum() > 200


@pytest.mark.parametrize("nx,ny,nz,num,nh", [(40, 44, 30, 2, 5), (34, 60, 30, 1, 7), (36, 64, 31, 3, 3)])
def test_split_windows(nx, ny, nz, num, nh):
    assert pct.query_plan(nx, ny, nz, num, nh)["groups"] > num
    v = volumes(nx, ny, nz, num, nx)
    with pct.Handle(0) as h:
        got = run(h, v, nh, pct.EXEC_B200_FP32)
    with pct.Handle(0) as h:
        h.set_memory_limit(4096)  # no partial sums: one item per tile
        ref = run(h, v, nh, pct.EXEC_B200_FP32)
    same(got, ref)


@pytest.mark.parametrize("nx,ny,nz,num,nh,k", [(40, 45, 30, 2, 7, 7), (36, 61, 30, 3, 7, 33), (38, 43, 33, 2, 9, 100)])
def test_prior_tiles(nx, ny, nz, num, nh, k):
    v = volumes(nx, ny, nz, num, nx + k)  # odd rows: tiles need the stacks repacked
    with pct.Handle(0) as h:
        h.set_learned_prior(k)
        got = run(h, v, nh, pct.EXEC_LEARNED)
    cap = 100_000
    while True:  # the least that the call runs with: no room for repacked stacks, so it rescores
        with pct.Handle(0) as h:
            h.set_learned_prior(k)
            h.set_memory_limit(cap)
            try:
                ref = run(h, v, nh, pct.EXEC_LEARNED)
                break
            except pct.PctError as e:
                assert e.status == -3
                cap += cap // 16
    same(got, ref)
