"""Ranks that share one device, in one launch without waits (algo local, the choice for emulated ranks): lengths
around the edges of packs, warps and tiles, aligned alike, misaligned alike, misaligned apart; blocks of
reduce_scatter and all_gather whose ragged length moves every block's alignment. Compared bit for bit with a plain PyTorch
reference that adds in fp32 in rank order and rounds once, as the kernel does; elements on both sides of every output must
stay as they were."""
import pytest
import torch

import nano_nccl_b200 as nn

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.float16, torch.bfloat16]
# one element; around a 16- and a 32-byte pack; a warp's packs; a tile's (8 ranks: 256 packs of 32 bytes) and more than one tile
COUNTS = [1, 7, 8, 9, 15, 16, 17, 255, 257, 511, 513, 2047, 2049, 4096, 4099, 16384 + 5, 70001]
PAD = 64


def buffers(ranks, numel, dtype, shifts, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    raw = [torch.full((numel + 2 * PAD,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
    views = [t[PAD + s:PAD + s + numel] for t, s in zip(raw, shifts)]
    if seed:
        for v in views:
            v.normal_(generator=gen)
    return raw, views


def untouched(raw, views):
    for t, v in zip(raw, views):
        lo = (v.data_ptr() - t.data_ptr()) // t.element_size()
        assert (t[:lo] == 7.0).all() and (t[lo + v.numel():] == 7.0).all()


def reference(ins, op):
    acc = ins[0].float()
    for t in ins[1:]:
        acc = acc + t.float() if op in ("sum", "avg") else (torch.maximum if op == "max" else torch.minimum)(acc, t.float())
    if op == "avg":
        acc = acc * torch.ones((), device="cuda").div(len(ins))  # 1/n in fp32, as the kernel takes it
    return acc.to(ins[0].dtype)


@pytest.mark.parametrize("ranks", range(2, 9))
@pytest.mark.parametrize("dtype", DTYPES)
def test_one_device_collectives_at_every_edge(ranks, dtype):
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, wait_timeout_ms=2000)
    try:
        half = 16 // torch.empty(0, dtype=dtype).element_size()  # 16 bytes: aligned alike modulo 16 only
        same, apart, halves = [1] * ranks, [r % 3 for r in range(ranks)], [half * (r % 2) + 1 for r in range(ranks)]
        for k, count in enumerate(COUNTS):
            op = ["sum", "avg", "max", "min"][k % 4]
            for shifts_in, shifts_out in (([0] * ranks, [0] * ranks), (same, same), ([0] * ranks, same), (same, [0] * ranks), (apart, apart), (halves, [0] * ranks)):
                _, ins = buffers(ranks, count, dtype, shifts_in, 100 + k)
                raw, outs = buffers(ranks, count, dtype, shifts_out, 0)
                comm.all_reduce(outs, ins, op=op)
                assert comm.last_call()["algo"] == "local"
                ref = reference(ins, op)
                for o in outs:
                    assert torch.equal(o, ref), (count, op, shifts_in, shifts_out)
                untouched(raw, outs)
                _, ins = buffers(ranks, count * ranks, dtype, shifts_in, 200 + k)
                raw, outs = buffers(ranks, count, dtype, shifts_out, 0)
                comm.reduce_scatter(outs, ins, op=op)
                ref = reference(ins, op)
                for r, o in enumerate(outs):
                    assert torch.equal(o, ref[r * count:(r + 1) * count]), (count, op, shifts_in, shifts_out)
                untouched(raw, outs)
                _, ins = buffers(ranks, count, dtype, shifts_in, 300 + k)
                raw, outs = buffers(ranks, count * ranks, dtype, shifts_out, 0)
                comm.all_gather(outs, ins)
                for o in outs:
                    assert torch.equal(o, torch.cat(ins)), (count, shifts_in, shifts_out)
                untouched(raw, outs)
        comm.check_async_error()
    finally:
        comm.close()


def test_in_place_on_one_device_and_a_capped_grid():
    comm = nn.Communicator(devices=[0], loopback_ranks=3, max_ctas=5, wait_timeout_ms=2000)
    try:
        for count in (17, 300003, 1 << 20):
            _, ins = buffers(3, count, torch.float32, [0, 0, 0], 9)
            ref = reference(ins, "sum")
            comm.all_reduce(ins)
            assert comm.last_call()["grid"] <= 5
            for t in ins:
                assert torch.equal(t, ref)
    finally:
        comm.close()


@pytest.mark.parametrize("ranks", [1, 8])
@pytest.mark.parametrize("cap", [1, 128, 160, 1000])
def test_a_cap_on_ctas_holds_at_any_value(ranks, cap):
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks if ranks > 1 else 0, max_ctas=cap, wait_timeout_ms=2000)
    try:
        for count in (1 << 20, (1 << 20) + 3):
            ins = [torch.full((count,), float(r + 1), device="cuda") for r in range(ranks)]
            for shift in (0, 1):  # 1: outputs that start one element past the inputs' alignment
                outs = [torch.zeros(count + 1, device="cuda")[shift:shift + count] for _ in range(ranks)]
                comm.all_reduce(outs, ins)
                torch.cuda.synchronize()
                assert 1 <= comm.last_call()["grid"] <= cap
                assert all((o == ranks * (ranks + 1) / 2).all() for o in outs)
        comm.check_async_error()
    finally:
        comm.close()


@pytest.mark.parametrize("ranks", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("collective", ["all_reduce", "reduce_scatter", "all_gather"])
def test_both_sizes_of_cta_around_their_tiles(ranks, collective):
    # 128 threads up to three CTAs for two SMs of what 256 would take, and in a reduce_scatter of four ranks and more; tiles of
    # 4096 or 2048 elements here (one rank: 16384 or 8192). Around that line and around a tile's end, three alignments.
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, wait_timeout_ms=2000) if ranks > 1 else nn.Communicator(devices=[0], wait_timeout_ms=2000)
    try:
        tile = 4096 if ranks > 1 else 16384
        segments = 1 if collective == "all_reduce" or ranks == 1 else ranks
        line = 222 // segments * tile
        for k, count in enumerate([line - tile - 1, line, line + 1, line + tile, line + tile + 2049, 3 * line + 16]):
            for s_in, s_out in ((0, 0), (1, 1), (0, 3)):
                n_in = count * (ranks if collective == "reduce_scatter" else 1)
                n_out = count * (ranks if collective == "all_gather" else 1)
                _, ins = buffers(ranks, n_in, torch.bfloat16, [s_in] * ranks, 500 + k)
                raw, outs = buffers(ranks, n_out, torch.bfloat16, [s_out] * ranks, 0)
                a, b = (outs, ins) if ranks > 1 else (outs[0], ins[0])
                if collective == "all_gather":
                    comm.all_gather(a, b)
                    expect = [torch.cat(ins)] * ranks
                else:
                    (comm.all_reduce if collective == "all_reduce" else comm.reduce_scatter)(a, b, op="avg")
                    full = reference(ins, "avg")
                    expect = [full] * ranks if collective == "all_reduce" else [full[r * count:(r + 1) * count] for r in range(ranks)]
                for o, e in zip(outs, expect):
                    assert torch.equal(o, e), (count, s_in, s_out)
                untouched(raw, outs)
    finally:
        comm.close()


@pytest.mark.parametrize("ranks", [1, 4, 8])
def test_a_cap_on_ctas_does_not_halve_their_threads(ranks):
    # CTAs of 128 threads are for calls that start as many of them as they like; a capped call whose CTAs loop keeps 256.
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks if ranks > 1 else 0, max_ctas=8, wait_timeout_ms=2000)
    try:
        for count, threads in ((2000, 128), ((1 << 17) + 3, 256)):
            ins = [torch.randn(count * ranks, device="cuda") for _ in range(ranks)]
            outs = [torch.empty(count, device="cuda") for _ in range(ranks)]
            full = [torch.empty(count * ranks, device="cuda") for _ in range(ranks)]
            if ranks == 1:
                comm.all_reduce(outs[0], ins[0])
                assert torch.equal(outs[0], ins[0])
            else:
                comm.reduce_scatter(outs, ins, op="max")
                most = torch.stack(ins).max(0).values
                assert all(torch.equal(o, most[r * count:(r + 1) * count]) for r, o in enumerate(outs))
                if threads == 256:
                    assert comm.last_call()["block"] == threads
                comm.all_gather(full, outs)
                assert all(torch.equal(f, most) for f in full)
                if threads == 256:
                    assert comm.last_call()["block"] == threads
                comm.all_reduce(full, ins, op="max")
                assert all(torch.equal(f, most) for f in full)
            info = comm.last_call()
            assert info["grid"] <= 8
            if threads == 256 or ranks == 1:
                assert info["block"] == threads, (count, info)
    finally:
        comm.close()
