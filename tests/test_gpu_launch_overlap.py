"""Kernels that start before their predecessor has ended must not lose by it."""
import pytest

from speedycolibri_b200 import synth
from speedycolibri_b200.configs import FMT_E4M3_ROW, MoeShape

pytestmark = pytest.mark.gpu


def test_the_three_launch_permutation_does_not_slow_the_expert_kernel(gpu_backend):
    """From 1024 (token, expert) pairs on the permutation takes three launches, whose last once let the
    register-level expert kernel start early: its CTAs packed onto the SMs that were free, and a call of 130
    tokens took 1.8 times one of 126.  Three per cent more tokens and two more launches stay within 1.3."""
    import torch

    from speedycolibri_b200.moe import Config, MoeBlock

    shape = MoeShape("overlap", H=2048, E=256, k=8, I=768, T=130, fmt=FMT_E4M3_ROW)
    blk = MoeBlock(Config.from_shape(shape), synth.device_layer(shape), 256)

    def best_of(T, rounds=5, calls=20):
        x = torch.randn((T, shape.H), device="cuda").to(torch.bfloat16)
        out = torch.empty_like(x)
        times = []
        for _ in range(rounds):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            blk.forward(x, out)
            begin.record()
            for _ in range(calls):
                blk.forward(x, out)
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)

    assert best_of(130) <= 1.3 * best_of(126)
    blk.close()
