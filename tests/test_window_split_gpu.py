"""Plans of the plain kernel that split the window's x offsets over CTAs (small volumes), on shapes
around the tiles' edges, against the FP64 oracle; with the memory cap and stream capture keeping a
plan to the scratch that there is."""
import numpy as np
import pytest
import torch

import oracle
import pseudoctimaging_b200 as pct
from conftest import compare_fused

pytestmark = pytest.mark.gpu

# (nx, ny, nz, num_atlas, nh): one interior voxel, one column, one tile and its neighbours (30 in
# y, 8 and 12 in x, 8..12 in z), prime atlas counts
SHAPES = [(13, 13, 13, 1, 11), (13, 44, 14, 2, 11), (21, 43, 21, 1, 11), (20, 42, 20, 3, 11),
          (22, 41, 23, 1, 9), (18, 40, 17, 5, 7), (17, 39, 20, 1, 7), (15, 37, 19, 2, 5),
          (16, 65, 13, 7, 3), (64, 64, 32, 1, 7)]


def run(h, s, lab, nh, div, stream=0):
    nz, nx, ny = s.img.shape
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (s.img, s.atlas_mri, lab)]
    out = torch.zeros_like(d[0])
    h.synthesize_device(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out.data_ptr(), nx, ny,
                        nz, s.atlas_mri.shape[0], nh, div, pct.EXEC_B200_FP32, stream)
    h.device_status(stream)
    return out.cpu().numpy()


@pytest.mark.parametrize("nx,ny,nz,num,nh", SHAPES)
def test_split_windows_match_oracle(nx, ny, nz, num, nh):
    plan = pct.query_plan(nx, ny, nz, num, nh)
    assert plan["groups"] > num, plan  # more groups than atlases: the window is split
    s = pct.synth_subject(nx, ny, nz, num, n_blobs=6, seed=nx + ny)
    lab = pct.normalize_labels(s.atlas_ct)
    div = pct.div_from(2.5, 1.0)
    with pct.Handle(0) as h:
        got = run(h, s, lab, nh, div)
        host = h.synthesize(s.img, s.atlas_mri, lab, nh, div)
    ref, prod, sumw = oracle.fuse_port(s.img, s.atlas_mri, lab, nh, div, with_sums=True)
    compare_fused(got, ref, nh, 1e-4, prod, sumw)
    np.testing.assert_array_equal(host, got)


def test_cap_and_capture_keep_to_the_scratch_there_is():
    nx, ny, nz, num, nh = 48, 40, 30, 2, 11
    s = pct.synth_subject(nx, ny, nz, num, n_blobs=6, seed=4)
    lab = pct.normalize_labels(s.atlas_ct)
    div = pct.div_from(2.5, 1.0)
    ref, prod, sumw = oracle.fuse_port(s.img, s.atlas_mri, lab, nh, div, with_sums=True)
    assert pct.query_plan(nx, ny, nz, num, nh)["scratch_bytes"] > 0
    with pct.Handle(0) as h:
        h.set_memory_limit(4096)  # the status word, no partial sums (ny % 4 == 0: no staging)
        compare_fused(run(h, s, lab, nh, div), ref, nh, 1e-4, prod, sumw)
    with pct.Handle(0) as h:
        t = pct.synth_subject(30, 32, 30, 1, n_blobs=4, seed=5)  # warm-up of a smaller volume
        run(h, t, pct.normalize_labels(t.atlas_ct), nh, div)
        d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (s.img, s.atlas_mri, lab)]
        out = torch.zeros_like(d[0])
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            h.synthesize_device(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out.data_ptr(),
                                nx, ny, nz, num, nh, div, pct.EXEC_B200_FP32,
                                torch.cuda.current_stream().cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        h.device_status()
        compare_fused(out.cpu().numpy(), ref, nh, 1e-4, prod, sumw)


def test_capture_after_a_warm_up_replays_the_same_plan():
    """A captured call whose scratch is there keeps its groups and their combine: the replay equals
    the direct call bit for bit, on new inputs in the same buffers too."""
    nx, ny, nz, num, nh = 40, 43, 26, 2, 9  # ny % 4 != 0: the repack is captured as well
    div = pct.div_from(2.5, 1.0)
    subs = [pct.synth_subject(nx, ny, nz, num, n_blobs=6, seed=k) for k in (6, 7)]
    labs = [pct.normalize_labels(s.atlas_ct) for s in subs]
    assert pct.query_plan(nx, ny, nz, num, nh)["groups"] > 1
    with pct.Handle(0) as h:
        ref = [run(h, s, lab, nh, div) for s, lab in zip(subs, labs)]
        d = [torch.empty(a.shape, device="cuda") for a in (subs[0].img, subs[0].atlas_mri, labs[0])]
        out = torch.zeros_like(d[0])
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            h.synthesize_device(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out.data_ptr(),
                                nx, ny, nz, num, nh, div, pct.EXEC_B200_FP32,
                                torch.cuda.current_stream().cuda_stream)
        for s, lab, r in zip(subs, labs, ref):
            for t, a in zip(d, (s.img, s.atlas_mri, lab)):
                t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
            g.replay()
            torch.cuda.synchronize()
            h.device_status()
            np.testing.assert_array_equal(out.cpu().numpy(), r)
