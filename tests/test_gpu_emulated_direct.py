"""One-shot and two-shot of emulated ranks (one launch, a CTA for every few KiB): buffers that are all misaligned alike, around
the packs and the CTAs' shares, for every rank count; bit for bit against a sum in rank order in fp32, rounded once."""
import pytest
import torch

import nano_nccl_b200 as nn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["oneshot", "twoshot"])
@pytest.mark.parametrize("ranks", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_buffers_misaligned_alike(algo, ranks, dtype):
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo=algo, wait_timeout_ms=2000)
    try:
        esz = torch.empty(0, dtype=dtype).element_size()
        gen = torch.Generator(device="cuda").manual_seed(ranks)
        share = 8192 // esz  # what one CTA of 256 threads takes at a time
        counts = [1, 16 // esz, 32 // esz, 48 // esz - 1, 62 // esz, 64 // esz + 1, 257, share * ranks - 1, share * ranks + 33, 3 * share * ranks + 5]
        for k, count in enumerate(counts):
            for shift in (1, 5, 16 // esz + 1, 32 // esz - 1):
                op = ["sum", "avg", "max", "min"][(k + shift) % 4]
                ins = [torch.randn(count + 64, device="cuda", generator=gen).to(dtype)[shift:shift + count] for _ in range(ranks)]
                raw = [torch.full((count + 64,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
                outs = [t[shift:shift + count] for t in raw]
                if algo == "twoshot" and k % 2:  # in place
                    for t, o in zip(ins, outs):
                        o.copy_(t)
                    comm.all_reduce(outs, outs, op=op)
                else:
                    comm.all_reduce(outs, ins, op=op)
                assert comm.last_call()["algo"] == algo
                acc = ins[0].float()
                for t in ins[1:]:
                    acc = acc + t.float() if op in ("sum", "avg") else (torch.maximum if op == "max" else torch.minimum)(acc, t.float())
                if op == "avg":
                    acc = acc * torch.tensor(1.0, device="cuda").div(ranks)
                expect = acc.to(dtype)
                for t, o in zip(raw, outs):
                    assert torch.equal(o, expect), (count, shift, op)
                    assert (t[:shift] == 7.0).all() and (t[shift + count:] == 7.0).all(), (count, shift, op)
        comm.check_async_error()
    finally:
        comm.close()


@pytest.mark.parametrize("algo", ["oneshot", "twoshot"])
def test_buffers_misaligned_differently_and_a_capped_grid(algo):
    # Not all alike modulo 16: element by element. And CTAs that loop, where the caller caps their number.
    comm = nn.Communicator(devices=[0], loopback_ranks=3, algo=algo, max_ctas=2, wait_timeout_ms=2000)
    try:
        gen = torch.Generator(device="cuda").manual_seed(5)
        for shifts, count in (((1, 2, 3), 30001), ((1, 1, 1), 100003), ((8, 8, 8), 100000), ((0, 0, 8), 4099)):
            ins = [torch.randn(count + 16, device="cuda", generator=gen).bfloat16()[s:s + count] for s in shifts]
            outs = [torch.zeros(count + 16, device="cuda", dtype=torch.bfloat16)[s:s + count] for s in shifts]
            comm.all_reduce(outs, ins)
            assert comm.last_call()["grid"] <= 2
            expect = (ins[0].float() + ins[1].float() + ins[2].float()).bfloat16()
            for o in outs:
                assert torch.equal(o, expect), (shifts, count)
    finally:
        comm.close()


@pytest.mark.parametrize("ranks", [2, 3, 8])
def test_low_latency_batches_of_words(ranks):
    # One word per thread at a time up to 16 KiB (32 KiB up to five ranks), four above: both sides of that line, a ragged batch, and
    # the largest message;
    # long and short messages in turn, so that slots of both kinds of call are used again.
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo="ll", wait_timeout_ms=2000)
    try:
        gen = torch.Generator(device="cuda").manual_seed(3)
        for k, words in enumerate([4096, 4097, 5, 8192, 8193, 16384, 16385, 4095, 16383, 32768, 1, 32767, 12289]):
            ins = [torch.randn(words * 2, device="cuda", generator=gen).half() for _ in range(ranks)]
            outs = [torch.empty_like(t) for t in ins]
            op = ["sum", "avg", "max", "min"][k % 4]
            comm.all_reduce(outs, ins, op=op)
            assert comm.last_call()["algo"] == "ll"
            acc = ins[0].float()
            for t in ins[1:]:
                acc = acc + t.float() if op in ("sum", "avg") else (torch.maximum if op == "max" else torch.minimum)(acc, t.float())
            if op == "avg":
                acc = acc * torch.tensor(1.0, device="cuda").div(ranks)
            for o in outs:
                assert torch.equal(o, acc.half()), (words, op)
        comm.check_async_error()
    finally:
        comm.close()


@pytest.mark.parametrize("ranks", [2, 8])
@pytest.mark.parametrize("rotate", [0, 1])
def test_low_latency_outputs_that_are_inputs(ranks, rotate):
    # In place, or into the next rank's input: a word is only overwritten when every rank has read it. Calls of both kinds in turn
    # share slots and counters.
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo="ll", wait_timeout_ms=2000)
    try:
        gen = torch.Generator(device="cuda").manual_seed(4)
        wrong = torch.zeros((), device="cuda", dtype=torch.int64)
        for k in range(60):
            words = (32768, 4096, 20000)[k % 3]
            ins = [torch.randn(words, device="cuda", generator=gen) for _ in range(ranks)]
            expect = torch.stack(ins).sum(0) if ranks == 2 else torch.stack(ins).max(0).values
            op = "sum" if ranks == 2 else "max"
            apart = [torch.empty_like(t) for t in ins]
            comm.all_reduce(apart, ins, op=op)
            outs = ins[rotate:] + ins[:rotate]
            comm.all_reduce(outs, ins, op=op)
            assert comm.last_call()["algo"] == "ll"
            for o in outs + apart:
                wrong += (o != expect).sum()
        assert wrong.item() == 0
        comm.check_async_error()
    finally:
        comm.close()


@pytest.mark.parametrize("algo", ["oneshot", "twoshot"])
@pytest.mark.parametrize("ranks", [2, 3, 8])
def test_ctas_that_loop_have_the_threads_of_a_whole_cta(algo, ranks):
    # A cap below what a call would take: 512 threads, shares of one, two and three rounds, and calls that read what the one before
    # wrote (the next launch may already wait on the SMs). Without a cap 256 threads.
    caps = {c: nn.Communicator(devices=[0], loopback_ranks=ranks, algo=algo, max_ctas=c, wait_timeout_ms=2000) for c in (2, 0)}
    try:
        gen = torch.Generator(device="cuda").manual_seed(11)
        parts = ranks if algo == "twoshot" else 1  # what the CTAs of a rank share: 8 KiB each without a cap
        for rounds in (2, 4, 5, 6):
            count = rounds * 2 * 4096 * parts + (3 if rounds == 5 else 0)
            for cap, comm in caps.items():
                ins = [torch.randn(count, device="cuda", generator=gen).bfloat16() for _ in range(ranks)]
                a, b = ([torch.zeros_like(t) for t in ins] for _ in range(2))
                comm.all_reduce(a, ins, op="avg")
                info = comm.last_call()
                assert info["algo"] == algo and info["block"] == (512 if cap else 256) and (not cap or info["grid"] == cap), info
                comm.all_reduce(b, a, op="max")
                comm.all_reduce(a, b, op="min")
                acc = ins[0].float()
                for t in ins[1:]:
                    acc = acc + t.float()
                expect = (acc * torch.tensor(1.0, device="cuda").div(ranks)).bfloat16()
                for o in a + b:
                    assert torch.equal(o, expect), (rounds, cap)
                blocks = [torch.zeros(count // ranks, device="cuda", dtype=torch.bfloat16) for _ in range(ranks)]
                whole = [torch.zeros(count // ranks * ranks, device="cuda", dtype=torch.bfloat16) for _ in range(ranks)]
                comm.reduce_scatter(blocks, [t[:count // ranks * ranks] for t in a], op="max")
                comm.all_gather(whole, blocks)
                for o in whole:
                    assert torch.equal(o, expect[:o.numel()]), (rounds, cap)
        for comm in caps.values():
            comm.check_async_error()
    finally:
        for comm in caps.values():
            comm.close()


@pytest.mark.parametrize("algo, cap", [("oneshot", 0), ("oneshot", 2), ("twoshot", 0), ("twoshot", 2), ("ll", 0)])
def test_captured_calls_follow_one_another(algo, cap):
    # Dependent launches as edges of a graph, with CTAs that loop and without; each call reads what the one before wrote.
    comm = nn.Communicator(devices=[0], loopback_ranks=4, algo=algo, max_ctas=cap, wait_timeout_ms=2000)
    try:
        count = 32768 if algo == "ll" else 300007
        ins = [torch.randn(count, device="cuda") for _ in range(4)]
        a, b, c = ([torch.empty_like(t) for t in ins] for _ in range(3))
        comm.all_reduce(a, ins, op="max")
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            comm.all_reduce(a, ins, op="max")
            comm.all_reduce(b, a, op="min")
            comm.all_reduce(c, b, op="max")
        for _ in range(5):
            for t in ins:
                t.normal_()
            graph.replay()
            torch.cuda.synchronize()
            expect = torch.stack(ins).max(0).values
            assert all(torch.equal(o, expect) for o in a + b + c)
        assert comm.last_call()["algo"] == algo
        comm.check_async_error()
    finally:
        comm.close()
