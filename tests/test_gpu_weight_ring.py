"""The tensor-memory expert kernel at the edges of its tiles and rings: row counts around the 16-row
granularity and the tile widths, feature counts that leave a partial 128-row tile (or no second one),
and contractions of an odd and an even number of k-tiles, in the three resident formats."""
import numpy as np
import pytest

from speedycolibri_b200 import synth
from speedycolibri_b200.configs import FMT_E4M3_ROW, FMT_FP8_B128, FMT_NVFP4, MoeShape
from tests.helpers import host_layer, upload_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [FMT_NVFP4, FMT_FP8_B128, FMT_E4M3_ROW], ids=["nvfp4", "fp8_b128", "e4m3_row"])
@pytest.mark.parametrize("H,I", [(264, 144), (1288, 400), (128, 128)])
@pytest.mark.parametrize("rows", [[1, 15, 16, 17, 33, 2, 64, 65], [159, 160, 161, 47, 1, 321]], ids=["short", "long"])
def test_tile_and_ring_edges(gpu_backend, orc, fmt, H, I, rows):
    shape = MoeShape("ring_edges", H=H, E=len(rows), k=1, I=I, T=4, fmt=fmt, shared=False, block_spread=1.0)
    L, packed = host_layer(shape)
    es = upload_layer(shape, packed).experts
    rng = np.random.default_rng(sum(rows))
    x = synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(rng.standard_normal((sum(rows), H)).astype(np.float32)))
    y = gpu_backend.expert_group([e.gate for e in es], [e.up for e in es], [e.down for e in es], rows, x)
    off = 0
    for e, r in enumerate(rows):
        want = L.expert_ffn(e, x[off:off + r])
        # h and y are rounded to bf16 (2^-9 relative each) and FP8 weights to f16 (2^-11): a row stays within 5e-3
        err = np.linalg.norm(y[off:off + r] - want, axis=1) / np.linalg.norm(want, axis=1)
        assert err.max() <= 5e-3, (e, r, err.max())
        off += r


@pytest.mark.parametrize("fmt", [FMT_NVFP4, FMT_FP8_B128, FMT_E4M3_ROW], ids=["nvfp4", "fp8_b128", "e4m3_row"])
def test_rows_past_the_end_of_a_tile_do_not_reach_the_results(gpu_backend, orc, fmt):
    """A partial weight tile leaves in the ring what the slot held before.  Every other expert of the group is
    all NaN, and a CTA's second tile is another expert's, one tile further: 3 tiles an expert, 240 in all."""
    rows_each, pairs = 9, 40
    shape = MoeShape("past_the_end", H=264, E=2, k=1, I=304, T=4, fmt=fmt, shared=False)
    L, packed = host_layer(shape)
    codes_or_scales = 1 if fmt == FMT_NVFP4 else 0
    for matrix in packed["experts"][0]:
        matrix[codes_or_scales][...] = 0x7F  # the NaN of e4m3
    nan, good = upload_layer(shape, packed).experts
    es = [nan, good] * pairs
    rng = np.random.default_rng(3)
    x = synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(rng.standard_normal((2 * pairs * rows_each, shape.H)).astype(np.float32)))
    y = gpu_backend.expert_group([e.gate for e in es], [e.up for e in es], [e.down for e in es], [rows_each] * len(es), x)
    y, x = (a.reshape(pairs, 2, rows_each, shape.H) for a in (y, x))
    assert np.isnan(y[:, 0]).all()
    want = L.expert_ffn(1, x[:, 1].reshape(-1, shape.H))
    got = y[:, 1].reshape(-1, shape.H)
    err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() <= 5e-3, err.max()  # the bound of the test above
