"""Plans of small volumes: no second round of the grid for a few items when a plan with as few rounds as
one takes less time (measured: 39 us against 47 for the first shape); and what planning itself costs."""
import time

import pytest
import torch

import pseudoctimaging_b200 as pct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(40, 23, 93, 8), (93, 10, 26, 14), (20, 118, 50, 10), (68, 16, 47, 10),
                                   (24, 48, 48, 14)])
def test_no_second_round_for_a_remainder(shape):
    p = pct.query_plan(*shape, 3)
    slots = pct.query_plan(222, 222, 112, 10, 11)["ctas"]  # a grid that is full
    rounds = p["groups"] * p["tiles"] / slots
    assert not 1 < rounds < 1.4, (rounds, p)


def test_the_prior_lists_its_offsets_once():
    """Sorting the window's offsets is most of a small call's host time (NH 11: 20 of 30 us): the centre
    prior's single offset, which does not run on tiles, takes 41 us with one sort and 63 with two."""
    d = [torch.rand(s, device="cuda") * 200 for s in ((40, 64, 64), (1, 40, 64, 64), (1, 40, 64, 64))]
    out = torch.zeros(40, 64, 64, device="cuda")

    def host_us(k):
        times = []
        with pct.Handle(0) as h:
            h.set_learned_prior(k)
            for _ in range(200):
                torch.cuda.synchronize()
                t = time.perf_counter()
                h.synthesize_device(*(x.data_ptr() for x in d), out.data_ptr(), 64, 64, 40, 1, 11, 337.5,
                                    pct.EXEC_LEARNED)
                times.append(1e6 * (time.perf_counter() - t))
        return sorted(times)[50]

    one, tiles = host_us(1), host_us(7)
    assert one < 1.75 * tiles, (one, tiles)
