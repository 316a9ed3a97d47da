"""The device-pointer calls of a handle refuse rows off the 16-byte grid before anything is launched: their
kernels read and write them 16 bytes at a time, and a misaligned access would take the context with it."""
import ctypes as C

import numpy as np
import pytest

from speedycolibri_b200 import _lib
from tests.fake_cuda import wrap_nvfp4

E, H, I, T, K = 4, 32, 16, 20, 2


@pytest.fixture(scope="module")
def handle(fake_cuda):
    tables = [(C.c_void_p * E)(*[wrap_nvfp4(fake_cuda, o, i) for _ in range(E)]) for o, i in ((I, H), (I, H), (H, I))]
    router = np.zeros((E, H), np.uint16)
    L = _lib.ColiMoeLayer(H=H, E=E, k=K, I=I, fmt=5, n_group=1, topk_group=1, ep_world=1, router_w=router.ctypes.data)
    L.gate, L.up, L.down = (C.cast(t, C.POINTER(C.c_void_p)) for t in tables)
    h = C.c_void_p()
    assert fake_cuda.coli_b200_moe_create(C.byref(h), C.byref(L), 64)
    return h


@pytest.mark.parametrize("call", ["block", "layer_step", "gather_local"])
@pytest.mark.parametrize("T", [1, 20], ids=["decode", "batch"])
def test_rows_off_the_16_byte_grid_are_refused(fake_cuda, handle, call, T):
    a, b = 0x7000000, 0x7800000  # stand-ins for device buffers: nothing reads them here

    def run(da, db):
        fake_cuda.fake_reset(0)
        x, y = C.c_void_p(a + da), C.c_void_p(b + db)
        if call == "block":
            ok = fake_cuda.coli_b200_moe_block_dev(handle, x, y, T, None)
        elif call == "layer_step":
            ok = fake_cuda.coli_b200_moe_layer_step_dev(handle, x, y, C.c_float(1e-5), T, None)
        else:
            ok = fake_cuda.coli_b200_moe_gather_local_dev(handle, x, C.c_void_p(b + 0x100000), T, y, C.c_void_p(b + 0x200000), C.c_void_p(b + 0x300000), None)
        return ok, fake_cuda.fake_queued()

    ok, queued = run(0, 0)
    assert ok == 1 and queued >= 1
    assert run(16, 48)[0] == 1
    for da, db in [(2, 0), (8, 0), (0, 2), (0, 8), (4, 4)]:
        assert run(da, db) == (0, 0), (da, db)
