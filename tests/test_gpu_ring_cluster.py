"""The ring of ranks that share a GPU (slices through distributed shared memory), at the edges of its rows of 32 vectors, its
slices of 1, 2, 4 and 8 rows, its windows and the rounds in which a warp takes them; every rank count; views that are misaligned
alike and differently; elements around every output must stay. Max and min are exact; a sum is off by at most one rounding of
the running sum per hop, so by ranks * 2^-24 (float32), 2^-11 (half) or 2^-8 (bfloat16) times the sum of the magnitudes."""
import ctypes

import pytest
import torch

import nano_nccl_b200 as nn
from nano_nccl_b200 import _lib

pytestmark = pytest.mark.gpu

EPS = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def check(got, ins, op, dtype):
    stack = torch.stack([t.float() for t in ins])
    if op in ("max", "min"):
        assert torch.equal(got.float(), (stack.max(0) if op == "max" else stack.min(0)).values), op
        return
    n = len(ins)
    ref, mag = stack.double().sum(0), stack.double().abs().sum(0)
    if op == "avg":
        ref, mag = ref / n, mag / n
    assert ((got.double() - ref).abs() <= 1.01 * (n + 1) * EPS[dtype] * mag + 1e-7).all(), op


@pytest.mark.parametrize("ranks", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("dtype", list(EPS))
def test_edges_of_rows_slices_and_windows(ranks, dtype):
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo="ring", wait_timeout_ms=2000)
    try:
        row = 512 // torch.empty(0, dtype=dtype).element_size()
        gen = torch.Generator(device="cuda").manual_seed(40 + ranks)

        def rand(count):
            return torch.randn(count, device="cuda", generator=gen).to(dtype)

        counts = [1, row - 1, row, row + 1, row * ranks, row * ranks + 1, 3 * row * ranks - 5, 700 * row * ranks + 3, 1500 * row * ranks - row,
                  5000 * row * ranks + 17]
        for k, count in enumerate(counts):
            for shifts in ([0] * ranks, [1] * ranks, [(r * 3) % 5 for r in range(ranks)]):
                op = ["sum", "max", "avg", "min"][(k + shifts[0]) % 4]
                ins = [rand(count + 8)[s:s + count] for s in shifts]
                raw = [torch.full((count + 40,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
                outs = [t[16 + s:16 + s + count] for t, s in zip(raw, shifts)]
                if op != "sum" and k % 2:  # in place
                    for o, t in zip(outs, ins):
                        o.copy_(t)
                    comm.all_reduce(outs, outs, op=op)
                else:
                    comm.all_reduce(outs, ins, op=op)
                assert comm.last_call()["algo"] == "ring"
                for t, o, s in zip(raw, outs, shifts):
                    check(o, ins, op, dtype)
                    assert torch.equal(o, outs[0])
                    assert (t[:16 + s] == 7.0).all() and (t[16 + s + count:] == 7.0).all(), (count, shifts)
            if count > 800 * row * ranks:
                continue
            big = [rand(count * ranks) for _ in range(ranks)]
            raw = [torch.full((count + 32,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
            shard = [t[16:16 + count] for t in raw]
            comm.reduce_scatter(shard, big, op=["max", "sum"][k % 2])
            for r in range(ranks):
                check(shard[r], [b[r * count:(r + 1) * count] for b in big], ["max", "sum"][k % 2], dtype)
                assert (raw[r][:16] == 7.0).all() and (raw[r][16 + count:] == 7.0).all()
            raw = [torch.full((count * ranks + 32,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
            full = [t[16:16 + count * ranks] for t in raw]
            comm.all_gather(full, shard)
            for t, o in zip(raw, full):
                assert torch.equal(o, torch.cat(shard))
                assert (t[:16] == 7.0).all() and (t[16 + count * ranks:] == 7.0).all()
        comm.check_async_error()
    finally:
        comm.close()


@pytest.mark.parametrize("ranks", [4, 8])
def test_slots_are_not_filled_before_they_are_read(ranks):
    # Every element names its place, so that a slice of another window or block shows. Slices of every call pass through the
    # same few slots; a slot returned too early was wrong in one of about 100 such calls.
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo="ring", wait_timeout_ms=2000)
    try:
        for count in (1 << 21, (1 << 21) + 5):
            ins = [(torch.arange(count, device="cuda", dtype=torch.int32) + r * count).view(torch.float32) for r in range(ranks)]
            expect = torch.cat(ins).view(torch.int32)
            outs = [torch.empty(count * ranks, device="cuda") for _ in range(ranks)]
            wrong = torch.zeros((), device="cuda", dtype=torch.int64)
            for _ in range(150):
                comm.all_gather(outs, ins)
                for o in outs:
                    wrong += (o.view(torch.int32) != expect).sum()
            assert wrong.item() == 0
        comm.check_async_error()
    finally:
        comm.close()


def test_nan_and_infinities_go_round():
    comm = nn.Communicator(devices=[0], loopback_ranks=4, algo="ring", wait_timeout_ms=2000)
    try:
        for dtype in EPS:
            ins = [torch.zeros(5000, device="cuda", dtype=dtype) for _ in range(4)]
            ins[1][17] = float("nan")
            ins[2][18] = float("inf")
            ins[3][4999] = -float("inf")
            for op in ("max", "min", "sum"):
                outs = [torch.empty_like(t) for t in ins]
                comm.all_reduce(outs, ins, op=op)
                for o in outs:
                    assert o[17].isnan() and o.isnan().sum() == 1, (dtype, op)
                    assert o[18] == (0.0 if op == "min" else float("inf")) and o[4999] == (0.0 if op == "max" else -float("inf"))
    finally:
        comm.close()


def test_a_cap_on_channels_and_calls_in_a_row_on_two_streams():
    comm = nn.Communicator(devices=[0], loopback_ranks=4, algo="ring", channels=3, wait_timeout_ms=2000)
    try:
        gen = torch.Generator(device="cuda").manual_seed(9)
        ins = [torch.randn(300007, device="cuda", generator=gen) for _ in range(4)]
        torch.cuda.synchronize()
        results, side = [], torch.cuda.Stream()
        for k in range(6):
            with torch.cuda.stream(side if k % 2 else torch.cuda.current_stream()):
                outs = [torch.empty_like(t) for t in ins]
                comm.all_reduce(outs, ins, op="max")
                assert comm.last_call()["grid"] <= 3
                results.append(outs)
        torch.cuda.synchronize()
        expect = torch.stack(ins).max(0).values
        assert all(torch.equal(o, expect) for outs in results for o in outs)
    finally:
        comm.close()


def test_wait_in_a_cluster_reports_instead_of_hanging():
    lib = _lib.load()
    out, waited = (ctypes.c_int * 4)(), ctypes.c_double()
    lib.b2_selftest_wait.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_double)]
    _lib.check(lib.b2_selftest_wait(2, 0, 50.0, out, ctypes.byref(waited)))
    assert out[0] == 0 and out[1] == 1 and out[2] == 97
    assert 45.0 <= waited.value <= 1000.0
    assert torch.ones(4, device="cuda").sum().item() == 4


@pytest.mark.parametrize("ranks", [2, 4, 8])
def test_slots_of_reducing_steps_are_not_filled_before_they_are_read(ranks):
    # As above for all_reduce and reduce_scatter, whose receiving steps also combine; with max every element names its place.
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo="ring", wait_timeout_ms=2000)
    try:
        for count in (1 << 20, (1 << 20) + 5):
            ins = [torch.arange(count, device="cuda", dtype=torch.float32) * ranks + (r + count) % ranks for r in range(ranks)]
            most = torch.stack(ins).max(0).values
            block = count // ranks
            outs = [torch.empty(count, device="cuda") for _ in range(ranks)]
            shards = [torch.empty(block, device="cuda") for _ in range(ranks)]
            parts = [t[:block * ranks] for t in ins]
            wrong = torch.zeros((), device="cuda", dtype=torch.int64)
            for _ in range(100):
                comm.all_reduce(outs, ins, op="max")
                comm.reduce_scatter(shards, parts, op="max")
                for o in outs:
                    wrong += (o != most).sum()
                wrong += (torch.cat(shards) != most[:block * ranks]).sum()
            assert wrong.item() == 0
        comm.check_async_error()
    finally:
        comm.close()


@pytest.mark.parametrize("channels", [1, 3, 32])
def test_a_channel_has_the_threads_of_a_whole_cta(channels):
    # A channel that somebody asks for is 512 threads of every rank, however many clusters make it up.
    comm = nn.Communicator(devices=[0], loopback_ranks=4, algo="ring", channels=channels, wait_timeout_ms=2000)
    try:
        for count in (1, 1 << 20, (1 << 22) + 3):
            ins = [torch.randn(count, device="cuda") for _ in range(4)]
            outs = [torch.empty_like(t) for t in ins]
            comm.all_reduce(outs, ins, op="max")
            info = comm.last_call()
            assert info["algo"] == "ring" and 1 <= info["grid"] <= channels and info["block"] == 512
            assert all(torch.equal(o, torch.stack(ins).max(0).values) for o in outs)
        assert info["grid"] == channels
    finally:
        comm.close()


def test_a_captured_ring():
    comm = nn.Communicator(devices=[0], loopback_ranks=4, algo="ring", wait_timeout_ms=2000)
    try:
        ins = [torch.randn(100003, device="cuda") for _ in range(4)]
        outs, again = ([torch.empty_like(t) for t in ins] for _ in range(2))
        comm.all_reduce(outs, ins, op="max")
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            comm.all_reduce(outs, ins, op="max")
            comm.all_reduce(again, outs, op="min")
        for _ in range(3):
            for t in ins:
                t.normal_()
            graph.replay()
            torch.cuda.synchronize()
            assert all(torch.equal(o, torch.stack(ins).max(0).values) for o in outs + again)
        comm.check_async_error()
    finally:
        comm.close()


def test_a_ring_in_clusters_takes_no_device_memory_for_fifos():
    def make():
        return nn.Communicator(devices=[0], loopback_ranks=4, algo="ring", wait_timeout_ms=2000)

    ins = [torch.randn(1 << 16, device="cuda") for _ in range(4)]
    outs = [torch.empty_like(t) for t in ins]
    first, second = make(), make()  # the first loads the kernels
    try:
        first.all_reduce(outs, ins, op="max")
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        second.all_reduce(outs, ins, op="max")
        torch.cuda.synchronize()
        assert free - torch.cuda.mem_get_info()[0] <= 4 << 20  # FIFOs in global memory would be 64 MiB
        assert all(torch.equal(o, torch.stack(ins).max(0).values) for o in outs)
        wires = second.ring_channel(1, 0)
        assert wires["send_fifo"] == wires["recv_fifo"] == 0 and wires["send_head"] != 0 and wires["recv_tail"] != 0
    finally:
        first.close()
        second.close()
