"""Two-shot of emulated ranks over host memory (transport shm), around its rows of 512 bytes, its growing and shrinking tiles and the
lines where the planner turns to the ring; views that start off a vector; every collective in turn on one communicator, so
that slots of one kind of call are used by the next. Sums are added in rank order in fp32 and rounded once: bit for bit."""
import pytest
import torch

import nano_nccl_b200 as nn

pytestmark = pytest.mark.gpu


def combine(ins, op):
    acc = ins[0].float()
    for t in ins[1:]:
        acc = acc + t.float() if op in ("sum", "avg") else (torch.maximum if op == "max" else torch.minimum)(acc, t.float())
    if op == "avg":
        acc = acc * torch.tensor(1.0, device="cuda").div(len(ins))
    return acc.to(ins[0].dtype)


@pytest.mark.parametrize("ranks", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_edges_of_rows_and_tiles(ranks, dtype):
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, transport="shm", wait_timeout_ms=3000)
    try:
        row = 512 // torch.empty(0, dtype=dtype).element_size()
        gen = torch.Generator(device="cuda").manual_seed(60 + ranks)

        def rand(count):
            return torch.randn(count, device="cuda", generator=gen).to(dtype)

        for k, count in enumerate([1, row - 1, row + 1, 15 * row * ranks, 16 * row * ranks + 3, 130 * row, 300 * row * ranks + row // 2, 1300 * row + 1]):
            for shift in (0, 1, 3):
                op = ["sum", "avg", "max", "min"][(k + shift) % 4]
                ins = [rand(count + 8)[shift:shift + count] for _ in range(ranks)]
                expect = combine(ins, op)
                raw = [torch.full((count + 40,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
                outs = [t[16 + shift:16 + shift + count] for t in raw]
                if k % 2:  # in place
                    for o, t in zip(outs, ins):
                        o.copy_(t)
                    comm.all_reduce(outs, outs, op=op)
                else:
                    comm.all_reduce(outs, ins, op=op)
                whole = comm.last_call()["algo"] == "twoshot"
                assert whole or ranks <= 3
                for t, o in zip(raw, outs):
                    assert not whole or torch.equal(o, expect), (count, shift, op)
                    assert (t[:16 + shift] == 7.0).all() and (t[16 + shift + count:] == 7.0).all(), (count, shift)
            for block in (count // ranks + 1, (count // ranks + 64) // 64 * 64):  # ragged, and whole vectors (the ring, where long)
                big = [rand(block * ranks) for _ in range(ranks)]
                raw = [torch.full((block + 32,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
                shards = [t[16:16 + block] for t in raw]
                comm.reduce_scatter(shards, big, op="max")
                for r in range(ranks):
                    assert torch.equal(shards[r], combine([b[r * block:(r + 1) * block] for b in big], "max")), block
                    assert (raw[r][:16] == 7.0).all() and (raw[r][16 + block:] == 7.0).all()
                raw = [torch.full((block * ranks + 32,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
                full = [t[16:16 + block * ranks] for t in raw]
                comm.all_gather(full, shards)
                for t, o in zip(raw, full):
                    assert torch.equal(o, torch.cat(shards)), block
                    assert (t[:16] == 7.0).all() and (t[16 + block * ranks:] == 7.0).all()
        torch.cuda.synchronize()
        comm.check_async_error()
    finally:
        comm.close()


def test_both_ways_of_one_communicator_in_a_captured_graph():
    # The first call takes the ring, the captured ones both: nothing is allocated while a stream is captured.
    comm = nn.Communicator(devices=[0], loopback_ranks=2, transport="shm", wait_timeout_ms=3000)
    try:
        long, short = [torch.randn(1 << 19, device="cuda") for _ in range(2)], [torch.randn(1000, device="cuda") for _ in range(2)]
        out_long, out_short = [torch.empty_like(t) for t in long], [torch.empty_like(t) for t in short]
        comm.all_reduce(out_long, long, op="max")
        assert comm.last_call()["algo"] == "ring"
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            comm.all_reduce(out_short, short, op="sum")
            assert comm.last_call()["algo"] == "twoshot"
            comm.all_reduce(out_long, long, op="max")
        for k in range(3):
            for t in long + short:
                t.normal_()
            graph.replay()
            torch.cuda.synchronize()
            assert all(torch.equal(o, torch.maximum(*long)) for o in out_long) and all(torch.equal(o, short[0] + short[1]) for o in out_short)
        comm.check_async_error()
    finally:
        comm.close()


def test_channels_asked_for_mean_a_ring():
    comm = nn.Communicator(devices=[0], loopback_ranks=4, transport="shm", channels=2, wait_timeout_ms=3000)
    try:
        ins = [torch.randn(1000, device="cuda") for _ in range(4)]
        outs = [torch.empty_like(t) for t in ins]
        comm.all_reduce(outs, ins, op="max")
        assert comm.last_call()["algo"] == "ring" and torch.equal(outs[3], combine(ins, "max"))
    finally:
        comm.close()
