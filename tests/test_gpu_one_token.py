"""One token, whose down projection and combine are one launch: formats, rows and K that end inside a tile, as many
rows and k-tiles as the launch takes and one more, and the residual stream of a layer step."""
import numpy as np
import pytest

from speedycolibri_b200 import synth
from speedycolibri_b200.configs import FMT_E4M3_ROW, FMT_FP8_B128, FMT_MXFP4, FMT_NVFP4, MoeShape
from tests.helpers import host_layer, rel_l2, upload_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [FMT_NVFP4, FMT_FP8_B128, FMT_E4M3_ROW, FMT_MXFP4], ids=["nvfp4", "fp8_b128", "e4m3_row", "mxfp4"])
@pytest.mark.parametrize("H,I,E,k,shared", [(264, 200, 20, 4, True), (128, 128, 20, 16, True), (72, 136, 20, 17, True),
                                            (128, 1032, 18, 17, False), (64, 8, 16, 1, False), (2368, 64, 8, 2, True), (2376, 64, 8, 2, True),
                                            (128, 896, 18, 4, True), (128, 904, 18, 4, True), (1800, 272, 20, 16, True)])
def test_one_token(gpu_backend, orc, fmt, H, I, E, k, shared):
    import torch

    from speedycolibri_b200 import _lib
    from speedycolibri_b200.moe import Config, MoeBlock

    shape = MoeShape("one_token", H=H, E=E, k=k, I=I, T=1, fmt=fmt, shared=shared, norm_topk=True)
    L, packed = host_layer(shape)
    blk = MoeBlock(Config.from_shape(shape), upload_layer(shape, packed), 1)
    x = synth.host_tokens(shape)
    before = _lib.load().coli_b200_launch_count()
    out, idx, w = blk.moe(x, want_routing=True)
    assert _lib.load().coli_b200_launch_count() - before == (3 if k + shared <= 17 and H <= 16 * 148 and I <= 7 * 128 else 4)
    want = L.moe_block(x)
    assert np.array_equal(idx, want["idx"]) and np.array_equal(w.view(np.uint32), want["w"].view(np.uint32))
    # h and y are rounded to bf16, 2^-9 relative each
    assert rel_l2(out, want["out"]) <= 5e-3

    rng = np.random.default_rng(H)
    resid = rng.standard_normal((1, H)).astype(np.float32)
    ln = (1.0 + 0.1 * rng.standard_normal(H)).astype(np.float32)
    step = synth.bf16_bits_to_f32(L.moe_block(synth.f32_to_bf16_bits(orc.rmsnorm(resid, ln, 1e-5)))["out"]).astype(np.float64)
    r = torch.from_numpy(resid.copy()).cuda()
    blk.layer_step(r, torch.from_numpy(ln).cuda(), 1e-5)
    delta = r.cpu().numpy().astype(np.float64) - resid
    assert np.linalg.norm(delta - step) <= 5e-3 * np.linalg.norm(step)
    blk.close()
