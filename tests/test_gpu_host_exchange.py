"""Two-shot of emulated ranks over host memory (transport shm), around its rows of 512 bytes, its growing and shrinking tiles and the
lines where the planner turns to the ring; views that start off a vector; every collective in turn on one communicator, so
that slots of one kind of call are used by the next. Sums are added in rank order in fp32 and rounded once: bit for bit."""
import os
import subprocess
import sys

import pytest
import torch

import nano_nccl_b200 as nn

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


SHM_CALLS = """
import torch, nano_nccl_b200 as nn
comm = nn.Communicator(devices=[0], loopback_ranks=4, transport="shm", algo=ALGO, wait_timeout_ms=3000)
ins = [torch.randn(1000, device="cuda") for _ in range(4)]
outs = [torch.empty_like(t) for t in ins]
comm.all_reduce(outs, ins, op="max")
assert all(torch.equal(o, torch.stack(ins).max(0).values) for o in outs)
comm.check_async_error()
print("ALGO", comm.last_call()["algo"])
comm.close()
"""


@pytest.mark.parametrize("algo, env, expect", [
    ("auto", {}, "twoshot"),
    ("ring", {}, "ring"),
    ("auto", {"B200CCL_RING_TURNAROUND": "1"}, "ring"),
    ("auto", {"B200CCL_RING_TURNAROUND": "0"}, "twoshot"),
    ("auto", {"B200CCL_FIFO_BUFF_BYTES": "1M"}, "ring"),
    ("auto", {"NANO_NCCL_FIFO_BUFF_BYTES": "1M"}, "ring"),
])
def test_what_only_a_ring_has_means_a_ring_and_no_other_memory(algo, env, expect):
    # The ring by name, its statistics or the size of its FIFOs: the ring runs, the statistics count its slices, and the up to 37 MiB of
    # host memory of the other way are not allocated.
    full = dict(os.environ, PYTHONPATH=ROOT, B200CCL_DEBUG="INFO", **env)
    p = subprocess.run([sys.executable, "-c", f"ALGO = {algo!r}\n" + SHM_CALLS], env=full, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                       timeout=240)
    assert p.returncode == 0 and f"ALGO {expect}" in p.stdout, p.stdout
    assert ("host exchange:" in p.stdout) == (expect == "twoshot"), p.stdout
    if env.get("B200CCL_RING_TURNAROUND") == "1":
        slices = [int(line.split(" slices=")[1].split()[0]) for line in p.stdout.splitlines() if line.startswith("ring turnaround")]
        assert len(slices) >= 4 and sum(slices) > 0, p.stdout


def algo_of(collective, ranks, bytes_, wide, aligned):
    # The lines of the planner, written out once more (bytes of the message, or of a block).
    if not wide and not (collective == "all_reduce" and aligned):
        return "twoshot"
    most = {"all_reduce": {2: 512 << 10, 3: 1 << 20}.get(ranks), "all_gather": 128 << 10 if ranks < 4 else None,
            "reduce_scatter": {2: 4 << 10, 8: 128 << 10}.get(ranks, 32 << 10)}[collective]
    return "twoshot" if most is None or bytes_ <= most else "ring"


@pytest.mark.parametrize("ranks", [2, 3, 4, 7, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_each_way_is_taken_where_the_planner_draws_the_line_and_is_right(ranks, dtype):
    # Both sides of every line, aligned and not: the expected algorithm runs; max is exact in both; sums bit for bit in two-shot and within
    # one rounding per hop in the ring.
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, transport="shm", wait_timeout_ms=3000)
    eps = {torch.float32: 2.0 ** -24, torch.bfloat16: 2.0 ** -8}[dtype]
    esz = torch.empty(0, dtype=dtype).element_size()
    gen = torch.Generator(device="cuda").manual_seed(70 + ranks)

    def compare(got, ins, op, algo):
        if algo == "twoshot" or op == "max":
            assert torch.equal(got, combine(ins, op))
        else:
            stack = torch.stack([t.double() for t in ins])
            assert ((got.double() - stack.sum(0)).abs() <= 1.01 * (ranks + 1) * eps * stack.abs().sum(0) + 1e-7).all()

    try:
        seen = set()
        for size in (4 << 10, 32 << 10, 128 << 10, 512 << 10, 1 << 20):
            for extra in (0, 16):
                for shift in (0, 1):
                    count = (size + extra) // esz
                    aligned = shift == 0
                    for op in ("sum", "max"):
                        ins = [torch.randn(count + shift, device="cuda", generator=gen).to(dtype)[shift:] for _ in range(ranks)]
                        outs = [torch.empty(count + shift, device="cuda", dtype=dtype)[shift:] for _ in range(ranks)]
                        comm.all_reduce(outs, ins, op=op)
                        algo = algo_of("all_reduce", ranks, count * esz, aligned, aligned)
                        seen.add(algo)
                        assert comm.last_call()["algo"] == algo, (size, extra, shift)
                        for o in outs:
                            compare(o, ins, op, algo)
                        whole = [torch.randn(count * ranks + shift, device="cuda", generator=gen).to(dtype)[shift:] for _ in range(ranks)]
                        comm.reduce_scatter(outs, whole, op=op)
                        algo = algo_of("reduce_scatter", ranks, count * esz, aligned, aligned)
                        assert comm.last_call()["algo"] == algo, (size, extra, shift)
                        for r, o in enumerate(outs):
                            compare(o, [t[r * count:(r + 1) * count] for t in whole], op, algo)
                        comm.all_gather(whole, outs)
                        assert comm.last_call()["algo"] == algo_of("all_gather", ranks, count * esz, aligned, aligned), (size, extra, shift)
                        assert all(torch.equal(t, torch.cat(outs)) for t in whole)
        assert "twoshot" in seen and (ranks > 3 or "ring" in seen)
        comm.check_async_error()
    finally:
        comm.close()
