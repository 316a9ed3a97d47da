"""Which result buffers of a host block call the last kernel writes itself: by the copies that the call queues."""
import ctypes as C

import numpy as np
import pytest

from speedycolibri_b200 import _lib
from tests.fake_cuda import wrap_nvfp4

E, H, I, T, K = 4, 32, 16, 20, 2
READ, READ_WRITE = 1, 3


@pytest.mark.parametrize("length,access,direct", [(0, READ_WRITE, False), (T * H * 2, READ_WRITE, True), (T * H * 2 - 1, READ_WRITE, False), (T * H * 2, READ, False)],
                         ids=["pageable", "pinned", "pinned_in_part", "pinned_read_only"])
def test_results_are_written_directly_only_where_the_device_may(fake_cuda, length, access, direct):
    tables = [(C.c_void_p * E)(*[wrap_nvfp4(fake_cuda, o, i)] * E) for o, i in ((I, H), (I, H), (H, I))]
    router = np.zeros((E, H), np.uint16)
    L = _lib.ColiMoeLayer(H=H, E=E, k=K, I=I, fmt=5, n_group=1, topk_group=1, ep_world=1, router_w=router.ctypes.data)
    L.gate, L.up, L.down = (C.cast(t, C.POINTER(C.c_void_p)) for t in tables)
    h = C.c_void_p()
    assert fake_cuda.coli_b200_moe_create(C.byref(h), C.byref(L), 64)
    x = np.zeros((T, H), np.uint16)
    room = np.zeros(T * H + 8, np.uint16)
    out = room[-room.ctypes.data % 16 // 2:][:T * H]  # on the 16-byte grid

    def queued(length, access):
        fake_cuda.fake_pin(C.c_void_p(out.ctypes.data), C.c_size_t(length), access)
        fake_cuda.fake_reset(0)
        assert fake_cuda.coli_b200_moe_block(h, x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p), T, None, None) == 1
        return fake_cuda.fake_queued()

    copied = queued(0, 0)
    assert queued(length, access) == copied - int(direct)
    fake_cuda.fake_pin(None, C.c_size_t(0), 0)
    fake_cuda.coli_b200_moe_destroy(h)
