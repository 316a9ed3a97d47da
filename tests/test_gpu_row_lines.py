"""Where a call moves from the register-level kernel to the tcgen05 kernel, on a layer of many weight tiles."""
import numpy as np
import pytest

from speedycolibri_b200 import _lib, synth
from speedycolibri_b200.configs import FMT_FP8_B128, FMT_NVFP4, MoeShape
from oracle.layers import oracle_layer_from_device

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
