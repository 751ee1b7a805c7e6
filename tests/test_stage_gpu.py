"""Host-pointer calls on pageable arrays (staged through pinned slots by worker threads) against the
same calls on pinned arrays (direct copies): identical outputs, for the overlapped and the one-upload
path, sizes that end in the middle of a slot, repeated calls, and two handles in two threads."""
import threading

import numpy as np
import pytest
import torch

import pseudoctimaging_b200 as pct

pytestmark = pytest.mark.gpu
DIV = 337.5


def volumes(nx, ny, nz, num, seed):
    g = torch.Generator().manual_seed(seed)
    base = torch.rand(nz, nx, ny, generator=g) * 400
    mri = base + torch.randn(num, nz, nx, ny, generator=g) * 3
    ct = torch.rand(num, nz, nx, ny, generator=g) * 2000 - 1000
    return [base + torch.randn(nz, nx, ny, generator=g) * 3, mri, ct]


def call(h, v, nh, choice, pipeline):
    a = [t.numpy() for t in v]
    if pipeline:
        return h.run_pipeline(*a, nh, 2.5, 1.0, choice, regularize=False)
    return h.synthesize(*a, nh, DIV, choice)


# (nx, ny, nz, num, nh, choice): overlapped uploads with and without the repack, one upload (one
# atlas; the centre prior), below the staging threshold
@pytest.mark.parametrize("nx,ny,nz,num,nh,choice", [
    (150, 141, 60, 4, 3, pct.EXEC_B200_FP32), (160, 128, 70, 5, 3, pct.EXEC_B200_FP32),
    (219, 203, 75, 1, 3, pct.EXEC_B200_FP32), (130, 127, 70, 3, 7, pct.EXEC_LEARNED),
    (40, 44, 30, 2, 5, pct.EXEC_B200_FP32)])
@pytest.mark.parametrize("pipeline", [False, True])
def test_pageable_equals_pinned(nx, ny, nz, num, nh, choice, pipeline):
    v = volumes(nx, ny, nz, num, nx)
    with pct.Handle(0) as h:
        if choice == pct.EXEC_LEARNED:
            h.set_learned_prior(7)
        ref = call(h, [t.pin_memory() for t in v], nh, choice, pipeline)
        for _ in range(2):  # the second call finds slots of the first
            got = call(h, v, nh, choice, pipeline)
            np.testing.assert_array_equal(got, ref)
        w = volumes(nx, ny, nz, num, nx + 1)
        other = call(h, w, nh, choice, pipeline)
        np.testing.assert_array_equal(other, call(h, [t.pin_memory() for t in w], nh, choice, pipeline))


def test_two_handles_in_two_threads():
    v = [volumes(150, 141, 60, 4, s) for s in (5, 6)]
    with pct.Handle(0) as h:
        refs = [call(h, x, 3, pct.EXEC_B200_FP32, False) for x in v]
    outs, errors = [None, None], []

    def work(k):
        try:
            with pct.Handle(0) as h:
                for _ in range(4):
                    outs[k] = call(h, v[k], 3, pct.EXEC_B200_FP32, False)
        except Exception as e:  # reported by the assertion below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for got, ref in zip(outs, refs):
        np.testing.assert_array_equal(got, ref)


def test_slots_pass_from_handle_to_handle():
    """Handles created and closed in turn, some alive at the same time, take over one another's
    pinned slots; after the last one is gone a new one starts afresh."""
    v = volumes(150, 141, 60, 4, 9)
    outs = []
    for _ in range(2):
        hs = [pct.Handle(0) for _ in range(4)]
        outs += [call(h, v, 3, pct.EXEC_B200_FP32, False) for h in hs]
        for h in hs[:3]:
            h.close()
        outs.append(call(hs[3], v, 3, pct.EXEC_B200_FP32, False))
        hs[3].close()
    for o in outs[1:]:
        np.testing.assert_array_equal(o, outs[0])


@pytest.mark.parametrize("ny,calls", [(141, 3), (212, 2)])
def test_slots_once_enough_was_copied(ny, calls):
    """41 MB calls copy directly first and through slots later, 62 MB calls through slots at once, on
    handles that come and go: the same volumes throughout."""
    v = volumes(136, ny, 60, 4, ny)
    with pct.Handle(0) as h:
        ref = call(h, [t.pin_memory() for t in v], 3, pct.EXEC_B200_FP32, False)
    for _ in range(2):
        a, b = pct.Handle(0), pct.Handle(0)
        for _ in range(calls):
            for h in (a, b):
                np.testing.assert_array_equal(call(h, v, 3, pct.EXEC_B200_FP32, False), ref)
        a.close()  # its slots go to the next handle
        with pct.Handle(0) as h:
            np.testing.assert_array_equal(call(h, v, 3, pct.EXEC_B200_FP32, False), ref)
        b.close()
