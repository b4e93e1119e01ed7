"""The kernels of real GPUs, asked for by name on one device (emulated ranks), at lengths around their packs: a message
that is no whole number of 16- or 32-byte packs leaves its last elements to single threads, misaligned buffers go
element by element. Compared with a plain PyTorch fp32 reference; elements around every output must stay."""
import pytest
import torch

import nano_nccl_b200 as nn

pytestmark = pytest.mark.gpu

TOL = {torch.float32: 1e-5, torch.float16: 2e-2, torch.bfloat16: 2e-1}


@pytest.mark.parametrize("algo", ["oneshot", "twoshot", "ll"])
@pytest.mark.parametrize("ranks", [2, 3, 8])
@pytest.mark.parametrize("dtype", list(TOL))
def test_peer_kernels_around_their_packs(algo, ranks, dtype):
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo=algo, wait_timeout_ms=2000)
    try:
        esz = torch.empty(0, dtype=dtype).element_size()
        counts = [1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 33, 255, 257, 1021, 4099, 65536 // esz - 1, 65536 // esz + 17]
        counts += [] if algo == "ll" else [300001]
        for k, count in enumerate(counts):
            if algo == "ll":
                count = -(-count * esz // 4) * 4 // esz  # whole words are all that it takes
            for shift in (0, 4 // esz):
                op = ["sum", "avg", "max", "min"][k % 4]
                gen = torch.Generator(device="cuda").manual_seed(700 + k)
                base = [torch.randn(count + 32, device="cuda", generator=gen).to(dtype) for _ in range(ranks)]
                ins = [t[16 + shift:16 + shift + count] for t in base]
                raw = [torch.full((count + 32,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
                outs = [t[16 + shift:16 + shift + count] for t in raw]
                comm.all_reduce(outs, ins, op=op)
                assert comm.last_call()["algo"] == algo
                stack = torch.stack([t.float() for t in ins])
                ref = {"sum": stack.sum(0), "avg": stack.sum(0) / ranks, "max": stack.max(0).values, "min": stack.min(0).values}[op]
                for t, o in zip(raw, outs):
                    assert (o.float() - ref).abs().max().item() <= TOL[dtype], (count, shift, op)
                    assert (t[:16 + shift] == 7.0).all() and (t[16 + shift + count:] == 7.0).all(), (count, shift)
                    assert torch.equal(o, outs[0])
        comm.check_async_error()
    finally:
        comm.close()


@pytest.mark.parametrize("ranks", [2, 3, 8])
@pytest.mark.parametrize("dtype", list(TOL))
def test_peer_reduce_scatter_and_all_gather_around_their_packs(ranks, dtype):
    # Blocks of every rank behind one another (reduce_kernel) and each rank's block into every output (gather_kernel): whole
    # packs, lengths that put every block on another alignment (4- and 2-byte accesses), buffers that start off a pack.
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo="oneshot", wait_timeout_ms=2000)
    try:
        esz = torch.empty(0, dtype=dtype).element_size()
        for k, block in enumerate([1, 2, 7, 8, 9, 16, 31, 256, 257, 1021, 4096, 4099, 65536 // esz, 65536 // esz + 2, 300001, 1 << 19]):
            for shift in (0, 1, 4 // esz):
                op = ["sum", "avg", "max", "min"][k % 4]
                gen = torch.Generator(device="cuda").manual_seed(800 + k)
                ins = [torch.randn(block * ranks + 32, device="cuda", generator=gen).to(dtype)[16 + shift:16 + shift + block * ranks] for _ in range(ranks)]
                raw = [torch.full((block + 64,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
                outs = [t[16 + shift:16 + shift + block] for t in raw]
                comm.reduce_scatter(outs, ins, op=op)
                assert comm.last_call()["algo"] == "oneshot"
                # added in rank order in fp32 and rounded once, so that a reference can match every bit
                acc = ins[0].float()
                for t in ins[1:]:
                    acc = acc + t.float() if op in ("sum", "avg") else (torch.maximum if op == "max" else torch.minimum)(acc, t.float())
                if op == "avg":
                    acc = acc * torch.tensor(1.0, device="cuda").div(ranks)
                expect = acc.to(dtype)
                for r, (t, o) in enumerate(zip(raw, outs)):
                    assert torch.equal(o, expect[r * block:(r + 1) * block]), (block, shift, op)
                    assert (t[:16 + shift] == 7.0).all() and (t[16 + shift + block:] == 7.0).all(), (block, shift)
                raw = [torch.full((block * ranks + 64,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
                full = [t[16 + shift:16 + shift + block * ranks] for t in raw]
                comm.all_gather(full, outs)
                assert comm.last_call()["algo"] == "oneshot"
                for t, o in zip(raw, full):
                    assert torch.equal(o, expect), (block, shift)
                    assert (t[:16 + shift] == 7.0).all() and (t[16 + shift + block * ranks:] == 7.0).all(), (block, shift)
        comm.check_async_error()
    finally:
        comm.close()
