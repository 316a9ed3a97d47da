"""From how many rows per segment on a block call takes the tcgen05 kernel: by the launchers that the call reaches."""
import ctypes as C

import numpy as np
import pytest

from speedycolibri_b200 import _lib
from speedycolibri_b200.configs import FMT_E4M3_ROW, FMT_FP8_B128, FMT_NVFP4
from tests.fake_cuda import wrap_nvfp4


def wrap(fake, fmt, O, I):
    if fmt == FMT_NVFP4:
        return wrap_nvfp4(fake, O, I)
    h = C.c_void_p()
    q, s = np.zeros((O, I), np.uint8), np.zeros(O * I, np.float32)
    fake.fake_reset(0)
    assert fake.coli_cuda_tensor_wrap(C.byref(h), q.ctypes.data_as(C.c_void_p), s.ctypes.data_as(C.c_void_p), fmt, I, O, 0)
    return h


# weight tiles of 128 features: E * ceil(I / 128); k pairs a token and no shared expert, so T * k / E rows per segment
@pytest.mark.parametrize("fmt,E,k,H,I,line", [
    (FMT_NVFP4, 40, 4, 256, 264, 10), (FMT_NVFP4, 111, 3, 256, 512, 10), (FMT_NVFP4, 89, 1, 256, 640, 9),        # 120, 444 | 445
    (FMT_NVFP4, 111, 3, 256, 1024, 9), (FMT_NVFP4, 127, 1, 256, 896, 8), (FMT_NVFP4, 120, 6, 128, 1920, 8),      # 888 | 889, one k-tile
    (FMT_FP8_B128, 40, 4, 256, 264, 8), (FMT_FP8_B128, 120, 6, 128, 1920, 8),
    (FMT_E4M3_ROW, 40, 4, 256, 264, 8), (FMT_E4M3_ROW, 120, 6, 128, 1920, 8),
])
def test_the_line_to_the_tcgen05_kernel(fake_cuda, fmt, E, k, H, I, line):
    # one handle stands for every expert
    tables = [(C.c_void_p * E)(*[wrap(fake_cuda, fmt, o, i)] * E) for o, i in ((I, H), (I, H), (H, I))]
    router = np.zeros((E, H), np.uint16)
    L = _lib.ColiMoeLayer(H=H, E=E, k=k, I=I, fmt=fmt, n_group=1, topk_group=1, ep_world=1, router_w=router.ctypes.data)
    L.gate, L.up, L.down = (C.cast(t, C.POINTER(C.c_void_p)) for t in tables)
    h = C.c_void_p()
    assert fake_cuda.coli_b200_moe_create(C.byref(h), C.byref(L), 16 * E)

    def kernel(T):
        fake_cuda.fake_reset(0)
        assert fake_cuda.coli_b200_moe_block_dev(h, C.c_void_p(0x7000000), C.c_void_p(0x7800000), T, None)
        names = fake_cuda.fake_launches().decode()
        assert ("launch_gate_up_tct" in names) != ("launch_gate_up_small" in names), names
        return "tcgen05" if "launch_gate_up_tct" in names else "decode"

    first = -(-line * E // k)  # the smallest T with line * E pairs
    assert (kernel(first - 1), kernel(first)) == ("decode", "tcgen05")
    fake_cuda.coli_b200_moe_destroy(h)
