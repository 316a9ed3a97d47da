"""Where a call moves from the register-level kernel to the tcgen05 kernel, on a layer of many weight tiles."""
import numpy as np
import pytest

from speedycolibri_b200 import _lib, synth
from speedycolibri_b200.configs import FMT_FP8_B128, FMT_NVFP4, MoeShape
from oracle.layers import oracle_layer_from_device, rel_l2

pytestmark = pytest.mark.gpu

EXPERTS, WIDTH = 120, 1920  # 120 x 15 tiles of 128 features: above the 1776 from which the block's line moves


@pytest.mark.parametrize("fmt", [FMT_NVFP4, FMT_FP8_B128], ids=["nvfp4", "fp8_b128"])
@pytest.mark.parametrize("rows_each,launches", [(6, 4), (7, 4), (8, 5)])
def test_host_group_below_eight_rows_writes_f32(gpu_backend, orc, fmt, rows_each, launches):
    """f32 -> f16, work list, gate+up, down; the tcgen05 kernels' bf16 result takes a fifth launch to f32."""
    shape = MoeShape("row_line", H=64, E=EXPERTS, k=1, I=WIDTH, T=4, fmt=fmt, shared=False)
    layer = synth.device_layer(shape)
    es = layer.experts
    x = np.random.default_rng(rows_each).standard_normal((EXPERTS * rows_each, shape.H)).astype(np.float32)
    before = _lib.load().coli_b200_launch_count()
    y = gpu_backend.expert_group([e.gate for e in es], [e.up for e in es], [e.down for e in es], [rows_each] * EXPERTS, x)
    assert _lib.load().coli_b200_launch_count() - before == launches
    rounded = (y.view(np.uint32) & 0xFFFF) == 0  # what bf16 holds; one value in 65536 by chance
    assert rounded.all() if launches == 5 else rounded.mean() < 0.01
    L = oracle_layer_from_device(shape, layer, {0, EXPERTS - 1})
    for e in (0, EXPERTS - 1):
        part = slice(e * rows_each, (e + 1) * rows_each)
        want = L.expert_ffn(e, x[part])
        # x in f16 (2^-12 relative), h in bf16 (2^-9) and from 8 rows on y too
        assert np.linalg.norm(y[part] - want) <= 5e-3 * np.linalg.norm(want)


@pytest.mark.parametrize("fmt,T,tcgen05", [(FMT_NVFP4, 119, False), (FMT_NVFP4, 120, True),
                                           (FMT_FP8_B128, 120, False), (FMT_FP8_B128, 159, False), (FMT_FP8_B128, 160, True)],
                         ids=["nvfp4_119", "nvfp4_120", "fp8_b128_120", "fp8_b128_159", "fp8_b128_160"])
def test_block_moves_at_six_rows_and_with_128x128_scales_at_eight(gpu_backend, orc, fmt, T, tcgen05):
    """6 experts of 120 per token: T / 20 rows per segment.  The tcgen05 kernel is given gathered rows, whose
    permutation takes three launches instead of one: router, top-k, permutation, gate+up, down, combine."""
    from speedycolibri_b200.moe import Config, MoeBlock

    shape = MoeShape("row_line_block", H=128, E=EXPERTS, k=6, I=WIDTH, T=T, fmt=fmt, shared=False)
    layer = synth.device_layer(shape)
    blk = MoeBlock(Config.from_shape(shape), layer, 256)
    x = synth.host_tokens(shape)
    before = _lib.load().coli_b200_launch_count()
    out, idx, _ = blk.moe(x, want_routing=True)
    assert _lib.load().coli_b200_launch_count() - before == (8 if tcgen05 else 6)
    sample = [0, T // 2, T - 1]
    want = oracle_layer_from_device(shape, layer, set(idx[sample].reshape(-1).tolist())).moe_block(x[sample])
    assert np.array_equal(idx[sample], want["idx"])
    # h and y in bf16 (2^-9 relative each), the 128x128 scales of the tcgen05 kernel in f16
    assert rel_l2(out[sample], want["out"]) <= 5e-3
    blk.close()
