"""The order in which the decode kernel adds an output's products is a function of the call's shapes: it depends neither
on where a row lies in the work list nor on what else is in the call."""
import numpy as np
import pytest

from speedycolibri_b200 import synth
from speedycolibri_b200.configs import FMT_E4M3_ROW, FMT_FP8_B128, FMT_NVFP4, MoeShape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [FMT_NVFP4, FMT_FP8_B128, FMT_E4M3_ROW], ids=["nvfp4", "fp8_b128", "e4m3_row"])
@pytest.mark.parametrize("experts,many", [(85, 60), (25, 17), (3, 9)], ids=["tasks_in_rounds", "less_than_a_round", "split_over_k"])
def test_a_row_gives_the_same_bits_wherever_it_lies(gpu_backend, fmt, experts, many):
    """One expert has `many` copies of a row, in several items of the list, the others have one row each; less than 8 rows
    an expert on average, so the results are f32.  With 85 experts the down launch has 92 items of 32 tasks on 148 SMs x
    16 or 18 warps: the copies' items lie on both sides of the end of its first round."""
    shape = MoeShape("sum_order", H=1024, E=experts, k=1, I=768, T=4, fmt=fmt, shared=False)
    es = synth.device_layer(shape).experts
    rng = np.random.default_rng(experts)
    rows = rng.standard_normal((experts, shape.H)).astype(np.float32)

    def call(order):
        counts = [many if e == order[at_copies] else 1 for e in order]
        x = np.concatenate([np.repeat(rows[e:e + 1], n, 0) for e, n in zip(order, counts)])
        y = gpu_backend.expert_group([es[e].gate for e in order], [es[e].up for e in order], [es[e].down for e in order], counts, x)
        ends = np.cumsum(counts)
        return {e: y[b - n:b].view(np.uint32) for e, n, b in zip(order, counts, ends)}

    at_copies = experts * 7 // 10
    order = list(range(experts))
    got = call(order)
    assert ((got[order[at_copies]] & 0xFFFF) != 0).any()  # f32 results
    assert all((y == y[:1]).all() for y in got.values())
    copied = order[at_copies]
    order.reverse()
    at_copies = order.index(copied)
    moved = call(order)
    assert all(np.array_equal(got[e], moved[e]) for e in order)
