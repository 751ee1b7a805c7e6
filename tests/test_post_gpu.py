"""Post-processing steps on the GPU against the reference's own outputs (through the C ABI):
NaN median fill (RegularizationStep), RoundMatrix + HU map, label normalisation, the FP64 error
reduction and the whole reference main() pipeline."""
import numpy as np
import pytest
import torch

import oracle
import pseudoctimaging_b200 as pct
from conftest import golden_names, load_golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def handle():
    h = pct.Handle(0)
    yield h
    h.close()


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("name", golden_names())
def test_regularize_matches_reference_bit_exact(handle, name):
    """Fed the reference's fused volume, the GPU fill reproduces RegularizationStep exactly."""
    g = load_golden(name)
    vol = torch.from_numpy(g["out"].copy()).cuda()
    nz, nx, ny = vol.shape
    fills = handle.regularize_device(vol.data_ptr(), nx, ny, nz, int(g["nh"]),
                                     torch.cuda.current_stream().cuda_stream)
    got = vol.cpu().numpy()
    assert np.array_equal(bits(got), bits(g["regularized"]))
    assert fills == int(np.isnan(g["out"]).sum())


@pytest.mark.parametrize("name", golden_names())
def test_finalize_hu_matches_reference_bit_exact(handle, name):
    g = load_golden(name)
    vol = torch.from_numpy(g["regularized"].copy()).cuda()
    handle.finalize_hu_device(vol.data_ptr(), vol.numel(), torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(bits(vol.cpu().numpy()), bits(g["hu"]))


def test_normalize_labels_matches_reference(handle):
    g = load_golden("nh9_3atlas")
    for offset in (0, 1):  # aligned and unaligned (scalar path) starts
        ct = torch.from_numpy(g["atlas_ct_hu"].reshape(-1).copy()).cuda()
        view = ct[offset:]
        handle.normalize_labels_device(view.data_ptr(), view.numel(),
                                       torch.cuda.current_stream().cuda_stream)
        assert np.array_equal(bits(view.cpu().numpy()), bits(g["label"].reshape(-1)[offset:]))


def test_error_stats_reduction(handle):
    g = load_golden("small_nh7_2atlas")
    a = g["out"].copy()
    b = g["out"].copy()
    lo = 4
    interior = (slice(lo, -lo),) * 3
    fin = np.argwhere(~np.isnan(a[interior]))
    z, x, y = fin[0] + lo
    a[z, x, y] += 2.0
    z2, x2, y2 = fin[1] + lo
    a[z2, x2, y2] = np.nan
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    nz, nx, ny = a.shape
    st = handle.error_stats_device(da.data_ptr(), db.data_ptr(), nx, ny, nz, 7,
                                   torch.cuda.current_stream().cuda_stream)
    n_fin = int((~np.isnan(b[interior])).sum())
    assert st["nan_mismatch"] == 1
    assert st["nan_both"] == int(np.isnan(b[interior]).sum())
    assert st["compared"] == n_fin - 1
    assert st["max_abs_hu"] == pytest.approx(2.0 * 4095 / 255, rel=1e-6)
    assert st["mae_hu"] == pytest.approx(2.0 * 4095 / 255 / (n_fin - 1), rel=1e-6)


@pytest.mark.parametrize("name", ["small_nh7_2atlas", "nan_rich_nh7", "nh9_3atlas"])
def test_pipeline_against_oracle_pipeline(handle, name):
    """normalise -> fuse -> regularise -> round -> HU, end to end on host buffers. The fused
    volume differs from FP64 in the last bits, so the HU output may differ by one rounding step
    (4095/255 ~ 16 HU) where a label value sits on a .5 boundary; no more than that."""
    g = load_golden(name)
    nh = int(g["nh"])
    got = handle.run_pipeline(g["img"], g["atlas_mri"], g["atlas_ct_hu"], nh, float(g["sigma"]),
                              float(g["beta"]))
    ref = g["hu"]
    assert not np.isnan(got).any()
    d = np.abs(got - ref)
    assert d.max() <= 17.0
    assert (d > 0).mean() < 0.01


def _sweep(vol, nh):
    """RegularizationStep in its sequential order on a copy (float64 median of float32 values)."""
    v = vol.copy()
    nz, nx, ny = v.shape
    lo = (nh - 1) // 2 + 1
    fills = 0
    for z, x, y in np.argwhere(np.isnan(v)):
        if lo <= z < nz - lo and lo <= x < nx - lo and lo <= y < ny - lo:
            n = v[z - 1:z + 2, x - 1:x + 2, y - 1:y + 2]
            n = n[~np.isnan(n)].astype(np.float64)
            v[z, x, y] = np.float32(np.median(n))
            fills += 1
    return v, fills


@pytest.mark.parametrize("shape,nh,holes", [((9, 9, 9), 7, 1), ((20, 33, 131), 3, 40),
                                            ((30, 40, 150), 11, 60), ((24, 70, 138), 5, 4000)])
def test_fill_follows_long_chains_in_sweep_order(handle, shape, nh, holes):
    """Boxes of NaN of up to 12 voxels a side (chains of dependent fills), rows that end before and
    after 128 columns, and lists longer than one voxel per warp: bit-exact."""
    r = np.random.default_rng(holes)
    nz, nx, ny = shape
    lo = (nh - 1) // 2 + 1
    vol = r.normal(50, 20, shape).astype(np.float32)
    for _ in range(holes):
        p = [int(r.integers(lo, n - lo)) for n in shape]
        e = [int(r.integers(1, 13)) if holes < 100 else int(r.integers(1, 5)) for _ in shape]
        vol[p[0]:p[0] + e[0], p[1]:p[1] + e[1], p[2]:p[2] + e[2]] = np.nan
    clean = np.nan_to_num(vol, nan=7.0)
    clean[lo:nz - lo, lo:nx - lo, lo:ny - lo] = vol[lo:nz - lo, lo:nx - lo, lo:ny - lo]
    ref, fills = _sweep(clean, nh)
    d = torch.from_numpy(clean).cuda()
    got_fills = handle.regularize_device(d.data_ptr(), nx, ny, nz, nh)
    assert np.array_equal(bits(d.cpu().numpy()), bits(ref))
    assert got_fills == fills


def test_fill_leaves_what_nothing_can_fill(handle):
    """NaN in the border may leave voxels without any value around them: the call ends and every
    voxel that a value reaches is filled."""
    vol = torch.full((11, 11, 11), float("nan"), device="cuda")
    assert handle.regularize_device(vol.data_ptr(), 11, 11, 11, 7) == 0
    assert bool(vol.isnan().all())
    vol[4, 4, 3] = 5.0  # a border value beside the first interior voxel
    assert handle.regularize_device(vol.data_ptr(), 11, 11, 11, 7) == 27
    assert bool((vol[4:7, 4:7, 4:7] == 5.0).all())
