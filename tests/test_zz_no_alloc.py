"""The allocation-free single-GPU all-reduce, called through its exported C symbol.

Some programs embedding the library may not allocate device memory when they need a reduction (all
memory already belongs to their own pool, or allocation is banned after start-up, or the stall of a
cudaMalloc is not acceptable at that point). ``b2_local_all_reduce_no_alloc`` serves them: one launch of
the one-device kernel, which needs no memory of its own. This test compares it, bit for bit, with a plain
PyTorch sum in fp32 in rank order, rounded once (the communicator's emulated ranks run the same kernel and
could not tell), on two calls in a row and on calls that overlap, and checks what it refuses with a
message. It is collected last on purpose (file name), so that a run that stops at the first failure has
already run every other test; it does not depend on any of them and also passes alone in a fresh process.
"""
import ctypes

import pytest
import torch

from nano_nccl_b200 import _lib

pytestmark = pytest.mark.gpu

DTYPE_CODE = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}
OP_CODE = {"sum": 0, "avg": 1, "max": 2, "min": 3}


def entry_point():
    lib = _lib.load()
    fn = lib.b2_local_all_reduce_no_alloc
    fn.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(ctypes.c_void_p), ctypes.c_int, ctypes.c_size_t,
                   ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    return lib, fn


def call(fn, inputs, outputs, op, status=None):
    n = len(inputs)
    ins = (ctypes.c_void_p * n)(*[t.data_ptr() for t in inputs])
    outs = (ctypes.c_void_p * n)(*[t.data_ptr() for t in outputs])
    stream = torch.cuda.current_stream().cuda_stream
    return fn(ins, outs, n, inputs[0].numel(), DTYPE_CODE[inputs[0].dtype], OP_CODE[op], stream,
              status.data_ptr() if status is not None else None)


def expected(inputs, op):
    acc = inputs[0].float()
    for t in inputs[1:]:
        acc = acc + t.float() if op in ("sum", "avg") else (torch.maximum if op == "max" else torch.minimum)(acc, t.float())
    if op == "avg":
        acc = acc * torch.ones((), device="cuda").div(len(inputs))  # 1/n in fp32, as the kernel takes it
    return acc.to(inputs[0].dtype)


@pytest.mark.parametrize("dtype,op,ranks,numel", [
    (torch.float32, "sum", 4, 1 << 20),     # many tiles
    (torch.bfloat16, "avg", 8, 4096),       # a few packs, fused 1/N
    (torch.float16, "max", 2, 65537),       # elements behind the last pack
    (torch.float32, "min", 1, 1000),        # a copy
])
def test_matches_a_plain_sum_on_two_calls_in_a_row(dtype, op, ranks, numel):
    torch.cuda.set_device(0)
    lib, fn = entry_point()
    status = torch.zeros(8, dtype=torch.int32, device="cuda")  # the 32-byte failure record: nothing waits, nothing is written
    for round_ in range(2):
        gen = torch.Generator(device="cuda").manual_seed(40 + round_)
        inputs = [torch.randn(numel, device="cuda", generator=gen).to(dtype) for _ in range(ranks)]
        got = [torch.full_like(t, float("nan")) for t in inputs]
        rc = call(fn, inputs, got, op, status)
        assert rc == 0, lib.b2_last_error()
        torch.cuda.synchronize()
        assert int(status.abs().sum().item()) == 0
        for g in got:
            assert torch.equal(g, expected(inputs, op))


def test_calls_on_two_streams_overlap_freely():
    torch.cuda.set_device(0)
    lib, fn = entry_point()
    streams = [torch.cuda.Stream() for _ in range(2)]
    sets = [[torch.randn(1 << 20, device="cuda") for _ in range(3)] for _ in range(6)]
    outs = [[torch.full_like(t, float("nan")) for t in s] for s in sets]
    torch.cuda.synchronize()
    for k, (s, o) in enumerate(zip(sets, outs)):
        with torch.cuda.stream(streams[k % 2]):
            assert call(fn, s, o, "sum") == 0, lib.b2_last_error()
    torch.cuda.synchronize()
    for s, o in zip(sets, outs):
        assert all(torch.equal(t, expected(s, "sum")) for t in o)


def test_rejects_what_it_cannot_reduce():
    torch.cuda.set_device(0)
    lib, fn = entry_point()
    x = [torch.zeros(16, device="cuda") for _ in range(9)]
    y = [torch.zeros(16, device="cuda") for _ in range(9)]
    assert call(fn, x, y, "sum") == 2
    msg = lib.b2_last_error().decode()
    assert "nranks = 9" in msg and "1..8" in msg
    assert call(fn, x[:2], x[:2], "sum") == 2 and b"in-place" in lib.b2_last_error()
    # ranges that overlap part-way, and two outputs that alias, would race inside the kernel
    big = torch.zeros(64, device="cuda")
    assert call(fn, [big[:16], big[32:48]], [big[8:24], big[48:64]], "sum") == 2 and b"overlap" in lib.b2_last_error()
    assert call(fn, x[:2], [big[:16], big[:16]], "sum") == 2 and b"outputs 0 and 1 overlap" in lib.b2_last_error()
    # a count whose byte size does not fit in size_t
    ins = (ctypes.c_void_p * 1)(x[0].data_ptr())
    outs = (ctypes.c_void_p * 1)(y[0].data_ptr())
    assert fn(ins, outs, 1, (1 << 63), 0, 0, None, None) == 2 and b"does not fit" in lib.b2_last_error()
    # and a valid call still works afterwards
    a = [torch.ones(16, device="cuda"), torch.full((16,), 2.0, device="cuda")]
    b = [torch.empty(16, device="cuda") for _ in range(2)]
    assert call(fn, a, b, "sum") == 0
    torch.cuda.synchronize()
    assert torch.equal(b[0], torch.full((16,), 3.0, device="cuda")) and torch.equal(b[1], b[0])
