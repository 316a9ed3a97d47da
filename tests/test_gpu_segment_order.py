"""Handles whose segment order is not expert order: the segments of an expert-parallel handle are sorted by
(owner, expert id), and one that holds every expert may still be called as a whole block."""
import numpy as np
import pytest

from speedycolibri_b200 import synth
from speedycolibri_b200.configs import CONFIGS
from speedycolibri_b200.moe import Config, MoeBlock
from tests.helpers import host_layer, rel_l2, upload_layer

pytestmark = pytest.mark.gpu


# 5 tokens: the decode front and the decode expert kernel; 37: the same behind the separate router and
# permutation; 433 and 333: the tcgen05 kernel, with and without a shared expert
@pytest.mark.parametrize("name,T", [("tiny", 5), ("tiny_sig", 37), ("mid", 433), ("mid_ragged", 333)])
@pytest.mark.parametrize("rank", [0, 1])
def test_whole_block_on_a_handle_with_alternating_owners(gpu_backend, orc, name, T, rank):
    import torch

    shape = CONFIGS[name].with_tokens(T)
    L, packed = host_layer(shape)
    blk = MoeBlock(Config.from_shape(shape), upload_layer(shape, packed), T, ep_rank=rank, ep_world=2,
                   expert_owner=[e % 2 for e in range(shape.E)])
    x = synth.host_tokens(shape, T)
    want = L.moe_block(x)
    # the bound of the same block on one GPU: h and y are rounded to bf16, 2^-9 relative each
    assert rel_l2(blk.moe(x), want["out"]) <= 5e-3
    out = blk.forward(torch.from_numpy(x.view(np.int16)).cuda().view(torch.bfloat16))
    assert rel_l2(out.view(torch.int16).cpu().numpy().view(np.uint16), want["out"]) <= 5e-3

    rng = np.random.default_rng(T)
    resid = rng.standard_normal((T, shape.H)).astype(np.float32)
    w = (1.0 + 0.1 * rng.standard_normal(shape.H)).astype(np.float32)
    step = synth.bf16_bits_to_f32(L.moe_block(synth.f32_to_bf16_bits(orc.rmsnorm(resid, w, 1e-5)))["out"]).astype(np.float64)
    r = torch.from_numpy(resid.copy()).cuda()
    blk.layer_step(r, torch.from_numpy(w).cuda(), 1e-5)
    blk.check()
    delta = r.cpu().numpy().astype(np.float64) - resid
    assert np.linalg.norm(delta - step) / np.linalg.norm(step) <= 5e-3
    blk.close()
