"""The centre prior on the plain kernel's tiles: every start of a tile's slab modulo 4 (the window's
half width moves it), runs of every length, sizes around the tiles' edges, unaligned rows, and the
rescoring where the memory cap leaves no room for the repacked stacks; against float64."""
import itertools

import numpy as np
import pytest

import pseudoctimaging_b200 as pct
from conftest import compare_fused
from test_learned_infer_gpu import DIV, fuse_offsets_f64, rows_of, subject

pytestmark = pytest.mark.gpu


def offsets(k, nh):
    h = (nh - 1) // 2
    return sorted(itertools.product(range(-h, h + 1), repeat=3),
                  key=lambda o: o[0] ** 2 + o[1] ** 2 + o[2] ** 2)[:k]


@pytest.mark.parametrize("nh,k", [(7, 2), (7, 7), (9, 7), (11, 7), (9, 20), (11, 33), (7, 81),
                                  (9, 100), (11, 124), (9, 125)])
@pytest.mark.parametrize("nx,ny,nz", [(21, 74, 23), (20, 43, 25), (33, 76, 19)])
def test_prior_runs_match_float64(nh, k, nx, ny, nz):
    num, lo = 2, (nh + 1) // 2
    img, atl, lab = subject(nx, ny, nz, num, nx + k)
    ref, prod, sumw = fuse_offsets_f64(img, atl, lab, offsets(k, nh), DIV, lo)
    with pct.Handle(0) as h:
        h.set_learned_prior(k)
        got = h.synthesize(img, atl, lab, nh, DIV, pct.EXEC_LEARNED)
        assert h.learned_stats() == {"fallback_pairs": 0,
                                     "row_offsets": rows_of(nx, ny, nz, lo) * k * num}
    compare_fused(got, ref, nh, 1e-4, prod, sumw)


def test_cap_without_room_for_the_repack_keeps_the_rescoring():
    import torch

    nx, ny, nz, num, nh, k = 22, 45, 24, 3, 11, 57
    img, atl, lab = subject(nx, ny, nz, num, 8)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (img, atl, lab)]
    outs = []
    for cap in (0, 1):
        with pct.Handle(0) as h:
            h.set_learned_prior(k)
            if cap:  # what the rescoring needs: found by a run that may not allocate anything more
                lim = 1 << 12
                while True:
                    h.set_memory_limit(lim)
                    try:
                        out = torch.zeros_like(d[0])
                        h.synthesize_device(*(t.data_ptr() for t in d), out.data_ptr(), nx, ny, nz,
                                            num, nh, DIV, pct.EXEC_LEARNED)
                        break
                    except pct.PctError as e:
                        assert e.status == -3
                        lim += lim // 8
            else:
                out = torch.zeros_like(d[0])
                h.synthesize_device(*(t.data_ptr() for t in d), out.data_ptr(), nx, ny, nz, num, nh,
                                    DIV, pct.EXEC_LEARNED)
            h.device_status()
            outs.append(out.cpu().numpy())
    ref, prod, sumw = fuse_offsets_f64(img, atl, lab, offsets(k, nh), DIV)
    for o in outs:
        compare_fused(o, ref, nh, 1e-4, prod, sumw)
