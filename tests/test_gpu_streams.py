"""Calls of one communicator on changing streams, on ONE device: a call sees what the call before it wrote on another
stream, waits for that call only and not for what the caller has queued behind it, and works while a blocking stream
is being captured elsewhere in the program."""
import time

import pytest
import torch

import nano_nccl_b200 as nn

pytestmark = pytest.mark.gpu


def communicator(ranks):
    return nn.Communicator(devices=[0], loopback_ranks=ranks if ranks > 1 else 0, wait_timeout_ms=2000)


@pytest.mark.parametrize("ranks", [1, 4])
@pytest.mark.parametrize("numel", [1024, 4 << 20])
def test_a_chain_of_calls_across_streams(ranks, numel):
    # Every call reads what the one before wrote; only the library orders the streams, which torch creates non-blocking.
    comm = communicator(ranks)
    try:
        steps = [None, torch.cuda.Stream(), None, torch.cuda.Stream(), torch.cuda.Stream(), None, None, torch.cuda.Stream()]
        chain = [[torch.full((numel,), 1.0 if k == 0 else float("nan"), device="cuda") for _ in range(ranks)] for k in range(len(steps) + 1)]
        torch.cuda.synchronize()
        for k, stream in enumerate(steps):
            comm.all_reduce(chain[k + 1], chain[k], op="sum", stream=stream)
        torch.cuda.synchronize()
        comm.check_async_error()
        for k, tensors in enumerate(chain):
            for t in tensors:
                assert (t == float(ranks ** k)).all(), k
    finally:
        comm.close()


def test_a_call_waits_for_the_call_before_and_nothing_else():
    comm = communicator(2)
    try:
        x = [torch.ones(1024, device="cuda") for _ in range(2)]
        y, z = [torch.empty_like(t) for t in x], [torch.empty_like(t) for t in x]
        side = torch.cuda.Stream()
        comm.all_reduce(y, x, stream=side)  # modules are loaded, tensors are there
        torch.cuda.synchronize()
        comm.all_reduce(y, x)
        torch.cuda._sleep(800_000_000)  # the caller's own work on the default stream, 0.4 s of it
        behind, done = torch.cuda.Event(), torch.cuda.Event()
        behind.record()
        comm.all_reduce(z, y, stream=side)
        done.record(side)
        while not done.query() and not behind.query():
            time.sleep(1e-3)
        independent = done.query() and not behind.query()
        torch.cuda.synchronize()
        comm.check_async_error()
        assert independent, "the call waited for work that was queued behind the previous call"
        assert (z[0] == 4.0).all() and (z[1] == 4.0).all()
    finally:
        comm.close()


@pytest.mark.parametrize("ranks", [1, 4])
def test_calls_while_a_blocking_stream_is_captured(ranks):
    rt = pytest.importorskip("cuda.bindings.runtime")
    comm = communicator(ranks)
    try:
        x = [torch.ones(4096, device="cuda") for _ in range(ranks)]
        y, z = [torch.empty_like(t) for t in x], [torch.empty_like(t) for t in x]
        side = torch.cuda.Stream()
        comm.all_reduce(y, x, stream=side)
        comm.all_reduce(y, x)  # the last call before the capture is on the default stream
        torch.cuda.synchronize()
        err, blocking = rt.cudaStreamCreate()
        assert err == rt.cudaError_t.cudaSuccess
        assert rt.cudaStreamBeginCapture(blocking, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)[0] == rt.cudaError_t.cudaSuccess
        failure = None
        try:
            comm.all_reduce(z, y, stream=side)
        except RuntimeError as e:
            failure = e
        ended, graph = rt.cudaStreamEndCapture(blocking)
        if ended == rt.cudaError_t.cudaSuccess:
            rt.cudaGraphDestroy(graph)
        rt.cudaGetLastError()
        rt.cudaStreamDestroy(blocking)
        torch.cuda.synchronize()
        assert failure is None and ended == rt.cudaError_t.cudaSuccess, (failure, ended)
        comm.check_async_error()
        assert all((t == float(ranks ** 2)).all() for t in z)
    finally:
        comm.close()
