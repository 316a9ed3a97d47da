"""The host expert call when one of its CUDA calls fails.  Copies from or to the caller's buffers and the
call's own tables may be queued by then, so on every path the last thing the call does to its stream is to
wait for it."""
import ctypes as C

import numpy as np
import pytest

from tests.fake_cuda import wrap_nvfp4


@pytest.mark.parametrize("rows", [3, 40], ids=["decode", "tcgen05"])
def test_a_host_group_call_that_fails_leaves_nothing_in_flight(fake_cuda, rows):
    H, I, count = 32, 16, 2
    tensors = [(C.c_void_p * count)() for _ in range(3)]
    for which, (o, i) in enumerate([(I, H), (I, H), (H, I)]):
        for c in range(count):
            tensors[which][c] = wrap_nvfp4(fake_cuda, o, i)
    n_rows = (C.c_int * count)(rows, rows)
    x, y = np.zeros((count * rows, H), np.float32), np.zeros((count * rows, H), np.float32)

    def call(fail_at):
        fake_cuda.fake_reset(fail_at)
        return fake_cuda.coli_cuda_expert_group_nvfp4(*tensors, n_rows, count, y.ctypes.data_as(C.c_void_p), x.ctypes.data_as(C.c_void_p))

    assert call(0) == 1 and fake_cuda.fake_waited()
    steps = fake_cuda.fake_queued()
    assert steps >= 10  # four events, three or more copies, three or more launches
    for n in range(1, steps + 1):
        assert call(n) == 0, n
        assert n == 1 or fake_cuda.fake_waited(), f"call {n} of {steps} on the stream failed and the call did not wait for those before it"
