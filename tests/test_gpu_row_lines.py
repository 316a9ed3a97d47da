"""Results on both sides of where a call moves from the decode kernel to the tcgen05 kernel (that it does is a CPU test's)."""
import numpy as np
import pytest

from speedycolibri_b200 import synth
from speedycolibri_b200.configs import FMT_FP8_B128, FMT_NVFP4, MoeShape
from oracle.layers import oracle_layer_from_device, rel_l2

pytestmark = pytest.mark.gpu

EXPERTS, WIDTH = 120, 1920  # 120 x 15 weight tiles of 128 features


@pytest.mark.parametrize("fmt", [FMT_NVFP4, FMT_FP8_B128], ids=["nvfp4", "fp8_b128"])
@pytest.mark.parametrize("rows_each,tcgen05", [(6, False), (7, False), (8, True)])
def test_host_group_below_eight_rows_writes_f32(gpu_backend, orc, fmt, rows_each, tcgen05):
    """The decode kernel writes f32, the tcgen05 kernel bf16 that is widened."""
    shape = MoeShape("row_line", H=64, E=EXPERTS, k=1, I=WIDTH, T=4, fmt=fmt, shared=False)
    layer = synth.device_layer(shape)
    es = layer.experts
    x = np.random.default_rng(rows_each).standard_normal((EXPERTS * rows_each, shape.H)).astype(np.float32)
    y = gpu_backend.expert_group([e.gate for e in es], [e.up for e in es], [e.down for e in es], [rows_each] * EXPERTS, x)
    rounded = (y.view(np.uint32) & 0xFFFF) == 0  # what bf16 holds; one value in 65536 by chance
    assert rounded.all() if tcgen05 else rounded.mean() < 0.01
    L = oracle_layer_from_device(shape, layer, {0, EXPERTS - 1})
    for e in (0, EXPERTS - 1):
        part = slice(e * rows_each, (e + 1) * rows_each)
        want = L.expert_ffn(e, x[part])
        # x in f16 (2^-12 relative), h in bf16 (2^-9) and from 8 rows on y too
        assert np.linalg.norm(y[part] - want) <= 5e-3 * np.linalg.norm(want)


# rows per segment around 6 and 8 on many weight tiles; 9 on 445 to 888; 10 on fewer
@pytest.mark.parametrize("fmt,H,E,k,I,T", [
    (FMT_NVFP4, 128, EXPERTS, 6, WIDTH, 119), (FMT_NVFP4, 128, EXPERTS, 6, WIDTH, 120),
    (FMT_NVFP4, 128, EXPERTS, 6, WIDTH, 159), (FMT_NVFP4, 128, EXPERTS, 6, WIDTH, 160),
    (FMT_FP8_B128, 128, EXPERTS, 6, WIDTH, 120), (FMT_FP8_B128, 128, EXPERTS, 6, WIDTH, 159), (FMT_FP8_B128, 128, EXPERTS, 6, WIDTH, 160),
    (FMT_NVFP4, 264, 90, 5, 640, 161), (FMT_NVFP4, 264, 90, 5, 640, 162),
    (FMT_NVFP4, 264, 40, 4, 264, 99), (FMT_NVFP4, 264, 40, 4, 264, 100),
])
def test_block_on_both_sides_of_its_lines(gpu_backend, orc, fmt, H, E, k, I, T):
    from speedycolibri_b200.moe import Config, MoeBlock

    shape = MoeShape("row_line_block", H=H, E=E, k=k, I=I, T=T, fmt=fmt, shared=False)
    layer = synth.device_layer(shape)
    blk = MoeBlock(Config.from_shape(shape), layer, 256)
    x = synth.host_tokens(shape)
    out, idx, _ = blk.moe(x, want_routing=True)
    sample = [0, T // 2, T - 1]
    want = oracle_layer_from_device(shape, layer, set(idx[sample].reshape(-1).tolist())).moe_block(x[sample])
    assert np.array_equal(idx[sample], want["idx"])
    # h and y in bf16 (2^-9 relative each), the 128x128 scales of the tcgen05 kernel in f16
    assert rel_l2(out[sample], want["out"]) <= 5e-3
    blk.close()
