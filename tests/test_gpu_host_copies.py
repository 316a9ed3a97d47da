"""Calls on pageable host memory against the same call on device memory, bit for bit: sizes on both sides of what goes
as it is, of a chunk of the page-locked ring, of its halves and of the whole of it."""
import ctypes
import mmap
import threading

import numpy as np
import pytest

from speedycolibri_b200 import synth
from speedycolibri_b200.configs import MoeShape

pytestmark = pytest.mark.gpu

H = 2048  # 4 KB a row


@pytest.fixture(scope="module")
def block(gpu_backend):
    from speedycolibri_b200.moe import Config, MoeBlock

    shape = MoeShape("host_copies", H=H, E=8, k=2, I=64, T=1, norm_topk=True)
    blk = MoeBlock(Config.from_shape(shape), synth.device_layer(shape), 1600)
    yield blk, shape
    blk.close()


def on_device(blk, x):
    import torch

    return blk.forward(torch.from_numpy(x.view(np.int16)).cuda().view(torch.bfloat16)).view(torch.int16).cpu().numpy().view(np.uint16)


@pytest.mark.parametrize("T", [1, 15, 16, 17, 63, 64, 65, 80, 511, 512, 513, 1024, 1025, 1536, 1537, 1600])
@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned"])
def test_host_rows_give_what_device_rows_give(block, T, pinned):
    import torch

    blk, shape = block
    x = synth.host_tokens(shape, T)
    want = on_device(blk, x)
    if pinned:
        src = torch.from_numpy(x.view(np.int16)).pin_memory()
        dst = torch.zeros((T, H), dtype=torch.int16).pin_memory()
        blk.moe_ptr(src.data_ptr(), dst.data_ptr(), T)
        got = dst.numpy().view(np.uint16)
    else:
        got = blk.moe(x)
    assert np.array_equal(got, want)


def test_host_calls_of_several_threads(block):
    blk, shape = block
    xs = [synth.host_tokens(shape, T, index=T) for T in (40, 300, 700, 1100)]
    want = [on_device(blk, x) for x in xs]
    bad = []

    def calls(i):
        for _ in range(5):
            if not np.array_equal(blk.moe(xs[i]), want[i]):
                bad.append(i)

    threads = [threading.Thread(target=calls, args=(i,)) for i in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_results_in_a_buffer_registered_in_parts(block):
    """Its first and last pages are page-locked, those between are not: it is copied to like any other."""
    from speedycolibri_b200 import _lib

    blk, shape = block
    x = synth.host_tokens(shape, 300)
    want = on_device(blk, x)
    page = mmap.PAGESIZE
    size = want.nbytes // page * page + 3 * page
    mem = mmap.mmap(-1, size)  # starts on a page
    out = np.frombuffer(mem, dtype=np.uint16, count=want.size)
    base = out.ctypes.data
    lib = _lib.load()
    parts = [base, base + (want.nbytes - 1) // page * page]
    assert all(lib.coli_cuda_host_register(ctypes.c_void_p(p), ctypes.c_size_t(page)) for p in parts)
    try:
        blk.moe_ptr(x.ctypes.data, base, 300)
        assert np.array_equal(out.reshape(want.shape), want)
    finally:
        for p in parts:
            lib.coli_cuda_host_unregister(ctypes.c_void_p(p))


@pytest.mark.parametrize("rows", [[1, 2, 4], [3, 4, 1], [2, 4, 3], [8, 8, 16], [9, 8, 16]])
def test_host_groups_on_both_sides_of_what_goes_as_it_is(gpu_backend, rows):
    """7, 8 and 9 rows of 8 KB below 8 an expert, 32 and 33 above: the rows of a call are those of calls with one row each."""
    shape = MoeShape("host_groups", H=H, E=3, k=1, I=64, T=1)
    es = synth.device_layer(shape).experts
    x = np.random.default_rng(sum(rows)).standard_normal((sum(rows), H)).astype(np.float32)
    y = gpu_backend.expert_group([e.gate for e in es], [e.up for e in es], [e.down for e in es], rows, x)
    of = np.repeat(np.arange(3), rows)
    for i in range(len(x)):
        want = gpu_backend.expert_group([es[of[i]].gate], [es[of[i]].up], [es[of[i]].down], [1], x[i:i + 1])[0]
        # h in bf16 on both sides, from 8 rows an expert on also y (2^-9 relative each)
        assert np.linalg.norm(y[i] - want) <= 5e-3 * np.linalg.norm(want)
