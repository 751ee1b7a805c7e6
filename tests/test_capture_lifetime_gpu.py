"""A captured call's scratch stays where the graph has it while its handle lives: later calls that need
more scratch, and other memory allocated in the meantime, change nothing about a replay."""
import numpy as np
import pytest
import torch

import pseudoctimaging_b200 as pct

pytestmark = pytest.mark.gpu
NH, DIV = 7, 337.5


def volumes(nx, ny, nz, num, seed):
    g = torch.Generator().manual_seed(seed)
    base = torch.rand(nz, nx, ny, generator=g) * 300
    d = [base + torch.randn(nz, nx, ny, generator=g) * 3,
         base + torch.randn(num, nz, nx, ny, generator=g) * 3, torch.rand(num, nz, nx, ny, generator=g) * 255]
    return [t.contiguous().cuda() for t in d] + [torch.zeros(nz, nx, ny, device="cuda")]


def call(h, d, choice):
    num, nz, nx, ny = d[1].shape
    h.synthesize_device(*(t.data_ptr() for t in d), nx, ny, nz, num, NH, DIV, choice,
                        torch.cuda.current_stream().cuda_stream)


# (small nx, ny, nz, num): a window split over CTAs, with and without the repack; the centre prior on
# stacks that are repacked for it
@pytest.mark.parametrize("small,choice", [((64, 64, 32, 1), pct.EXEC_B200_FP32),
                                          ((40, 43, 26, 2), pct.EXEC_B200_FP32),
                                          ((33, 45, 24, 2), pct.EXEC_LEARNED)])
def test_replay_after_larger_calls(small, choice):
    large = (150, 141, 60, 6)
    with pct.Handle(0) as h:
        if choice == pct.EXEC_LEARNED:
            h.set_learned_prior(33)
        else:
            assert 0 < pct.query_plan(*small, NH)["scratch_bytes"] < pct.query_plan(*large, NH)["scratch_bytes"]
        d, e = volumes(*small, 1), volumes(*small, 2)
        refs = []
        for v in (d, e):
            call(h, v, choice)
            torch.cuda.synchronize()
            refs.append(v[3].clone())
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call(h, d, choice)
        big = volumes(*large, 3)
        call(h, big, choice)
        torch.cuda.synchronize()
        first = big[3].clone()
        other = pct.Handle(0)  # takes what a closed handle may have left
        with pct.Handle(0) as closed:
            call(closed, volumes(*small, 4), pct.EXEC_B200_FP32)
        call(other, big, pct.EXEC_B200_FP32)
        filler = torch.full((64, 1 << 20), 7.0, device="cuda")
        for v, ref in zip((d, e), refs):
            for a, b in zip(d[:3], v[:3]):
                a.copy_(b)
            d[3].zero_()
            g.replay()
            torch.cuda.synchronize()
            h.device_status()
            np.testing.assert_array_equal(d[3].cpu().numpy(), ref.cpu().numpy())
        assert bool((filler == 7.0).all())
        big[3].zero_()
        call(h, big, choice)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(big[3].cpu().numpy(), first.cpu().numpy())
        other.close()


@pytest.mark.parametrize("mode", ["relaxed", "thread_local"])
def test_closing_a_handle_leaves_captures_alone(mode):
    """A handle with partial sums is closed (in another thread) while a stream is being captured."""
    import threading

    h = pct.Handle(0)
    d = volumes(64, 64, 32, 1, 5)
    call(h, d, pct.EXEC_B200_FP32)
    torch.cuda.synchronize()
    with pct.Handle(0):  # not the last handle: its partial sums are kept
        x = torch.zeros(16, device="cuda")
        g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.stream(s):
            g.capture_begin(capture_error_mode=mode)
            x.add_(1)
            t = threading.Thread(target=h.close)
            t.start()
            t.join()
            x.add_(1)
            g.capture_end()
        g.replay()
        torch.cuda.synchronize()
        assert float(x[0]) == 2.0


def test_sums_are_passed_on_only_when_idle():
    """A handle closed right after an asynchronous call: the next handle's call, which takes over the
    partial sums, waits for it."""
    d, e = volumes(64, 64, 32, 3, 6), volumes(64, 64, 32, 3, 7)
    assert 0 < pct.query_plan(64, 64, 32, 3, NH)["scratch_bytes"] <= 32 << 20
    refs = []
    for v in (d, e):
        with pct.Handle(0) as h:
            call(h, v, pct.EXEC_B200_FP32)
            torch.cuda.synchronize()
        refs.append(v[3].clone())
        v[3].zero_()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    with pct.Handle(0):
        for _ in range(10):
            for v, s in zip((d, e), streams):
                with torch.cuda.stream(s), pct.Handle(0) as h:
                    call(h, v, pct.EXEC_B200_FP32)
    torch.cuda.synchronize()
    for v, ref in zip((d, e), refs):
        np.testing.assert_array_equal(v[3].cpu().numpy(), ref.cpu().numpy())
