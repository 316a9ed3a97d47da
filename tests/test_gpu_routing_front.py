"""Router, top-k and permutation at the edges of their paths: the decode front (up to 8 tokens), the staged router
(8 x 8 tiles up to the number of SMs), rows placed by the counts of the top-k (with a copy of x and with gathered
rows, around 1024 pairs), and the selection by counting with more candidates than a warp has lanes."""
import numpy as np
import pytest

from speedycolibri_b200 import synth
from speedycolibri_b200.configs import SCORE_SIGMOID, SCORE_SOFTMAX, MoeShape
from oracle.layers import oracle_layer_from_device, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,k,H,score,groups,shared", [
    (1, 32, 1, 24, SCORE_SOFTMAX, 1, False), (1, 128, 8, 520, SCORE_SOFTMAX, 1, True), (8, 40, 32, 264, SCORE_SOFTMAX, 1, True),
    (7, 257, 8, 256, SCORE_SIGMOID, 1, True), (8, 512, 8, 1032, SCORE_SOFTMAX, 1, False), (3, 256, 8, 248, SCORE_SIGMOID, 8, True),
    (8, 96, 6, 136, SCORE_SIGMOID, 3, True), (2, 64, 4, 512, SCORE_SIGMOID, 32, False),                    # decode front
    (9, 70, 5, 64, SCORE_SIGMOID, 7, True), (32, 64, 8, 64, SCORE_SOFTMAX, 1, True), (33, 64, 8, 64, SCORE_SOFTMAX, 1, True),
    (256, 300, 1, 64, SCORE_SOFTMAX, 1, True), (32, 296, 8, 1032, SCORE_SOFTMAX, 1, False),                 # 148 tiles of the staged router
    (33, 296, 8, 520, SCORE_SIGMOID, 1, True), (130, 400, 8, 264, SCORE_SOFTMAX, 1, True),                  # ... 185 tiles; 1040 pairs, x copied
    (12, 4, 4, 264, SCORE_SOFTMAX, 1, True), (170, 20, 6, 264, SCORE_SOFTMAX, 1, True),                     # gathered: 31 KB | 1020 pairs, 628 KB
    (171, 20, 6, 264, SCORE_SOFTMAX, 1, True), (600, 512, 32, 72, SCORE_SIGMOID, 1, False),                 # 1026 and 19200 pairs
    (29, 20, 6, 264, SCORE_SOFTMAX, 1, True), (30, 20, 6, 264, SCORE_SOFTMAX, 1, True),                     # 9.7 | 10 rows a segment: two items each
    (2049, 40, 32, 24, SCORE_SOFTMAX, 1, True),                                                             # above 65536 pairs
])
@pytest.mark.parametrize("equal", [0, 40], ids=["distinct", "ties"])
def test_routing_and_block_at_the_edges(gpu_backend, orc, T, E, k, H, score, groups, shared, equal):
    from speedycolibri_b200.moe import Config, MoeBlock

    shape = MoeShape("front_edges", H=H, E=E, k=k, I=16, T=T, shared=shared, norm_topk=True, score=score, n_group=groups,
                     topk_group=max(1, (groups + 1) // 2), select_bias_std=0.0 if equal else 0.01)
    layer = synth.device_layer(shape)
    if equal:  # equal rows of the router give equal logits: ties go to the lowest id
        layer.router[:equal] = layer.router[0]
    blk = MoeBlock(Config.from_shape(shape), layer, max(T, 8))
    x = synth.host_tokens(shape)
    x[T // 2] = 0  # all logits of this token are equal
    out, idx, w = blk.moe(x, want_routing=True)
    L = oracle_layer_from_device(shape, layer, set(range(E)))
    want = L.moe_block(x)
    assert np.array_equal(idx, want["idx"])
    assert np.array_equal(w.view(np.uint32), want["w"].view(np.uint32))
    # h and y are rounded to bf16, 2^-9 relative each
    assert rel_l2(out, want["out"]) <= 5e-3
    blk.close()


@pytest.mark.parametrize("T", [12, 60, 170, 171])
def test_gathered_rows_are_placed_in_one_launch(gpu_backend, T):
    """72 to 1026 pairs, 44 KB to 632 KB of rows: router, top-k, placement, gate+up, down, combine."""
    import torch

    from speedycolibri_b200 import _lib
    from speedycolibri_b200.moe import Config, MoeBlock

    shape = MoeShape("front_launches", H=264, E=4 if T == 12 else 20 if T > 60 else 6, k=4 if T == 12 else 6, I=16, T=T)
    blk = MoeBlock(Config.from_shape(shape), synth.device_layer(shape), T)
    x = torch.randn((T, shape.H), device="cuda").to(torch.bfloat16)
    before = _lib.load().coli_b200_launch_count()
    blk.forward(x)
    assert _lib.load().coli_b200_launch_count() - before == 6
    torch.cuda.synchronize()
    blk.close()
