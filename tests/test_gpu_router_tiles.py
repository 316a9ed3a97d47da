"""Every tile of the router GEMM against the oracle's sequential logits, bit for bit: batches that end
inside a tile on both axes, hidden sizes that end inside a k-block, and rows off the 16-byte grid."""
import numpy as np
import pytest

from speedycolibri_b200 import _lib, synth
from speedycolibri_b200.configs import SCORE_SIGMOID, MoeShape

pytestmark = pytest.mark.gpu


TILES = ["8 x 8", "16 x 32", "64 x 64", "128 x 64", "128 x 128"]  # tokens x experts, by coli_b200_router_tile's number


@pytest.mark.parametrize("tile,T,E,H,offset", [
    ("8 x 8", 1, 9, 8, 0), ("8 x 8", 9, 130, 136, 0), ("8 x 8", 8, 128, 2048, 0),
    ("16 x 32", 610, 140, 200, 0),
    ("64 x 64", 2050, 250, 72, 0),
    ("128 x 64", 4000, 250, 72, 0),
    ("128 x 128", 9500, 380, 72, 0),
    (None, 20, 40, 136, 1),                                 # rows that are not 16-byte aligned
])
def test_router_tiles_bit_exact(gpu_backend, orc, tile, T, E, H, offset):
    import torch

    from speedycolibri_b200.moe import Config, MoeBlock

    if tile is not None:
        assert TILES[_lib.load().coli_b200_router_tile(T, E)] == tile  # the case still covers the tile it names
    shape = MoeShape("router_tiles", H=H, E=E, k=4, I=16, T=T, shared=False, norm_topk=True, score=SCORE_SIGMOID,
                     select_bias_std=0.01)
    layer = synth.device_layer(shape)
    blk = MoeBlock(Config.from_shape(shape), layer, T)
    xh = synth.host_tokens(shape)
    flat = torch.zeros(T * H + 8, dtype=torch.int16, device="cuda")
    x = flat[offset:offset + T * H].view(T, H)
    x.copy_(torch.from_numpy(xh.view(np.int16)))
    idx = torch.empty((T, shape.k), dtype=torch.int32, device="cuda")
    w = torch.empty((T, shape.k), dtype=torch.float32, device="cuda")
    blk.topk_dev(x, idx, w, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    L = orc.Layer(H, E, shape.k, shape.I, shape.score, shape.norm_topk, shape.routed_scale, 1, 1, shape.fmt, layer.router,
                  [None] * E, None, layer.router_bias, None)
    want_idx, want_w = L.route_tokens(xh)
    assert np.array_equal(idx.cpu().numpy(), want_idx)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), want_w.view(np.uint32))
    blk.close()
