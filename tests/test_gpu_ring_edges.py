"""Ring kernel on one device at the edges of its slice loop: slices of one batch (512 threads x 8 vectors) and a
vector or an element more or less, ragged messages whose last elements fill no vector, blocks that fall back to
single elements, several calls in a row. Compared with a plain PyTorch fp32 reference."""
import pytest
import torch

import nano_nccl_b200 as nn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ranks,channels", [(2, 1), (3, 2), (8, 16)])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 2e-1)])
@pytest.mark.parametrize("transport", ["auto", "shm"])
def test_ring_slices_at_the_edges(ranks, channels, dtype, tol, transport):
    comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo="ring", transport=transport, channels=channels, wait_timeout_ms=3000)
    try:
        vec = 16 // torch.empty(0, dtype=dtype).element_size()
        batch = 512 * 8 * vec
        base = 2 * ranks * channels * batch if channels < 16 else 4096 * vec
        for k, count in enumerate([1, vec + 1, 512 * vec * ranks, base - 1, base, base + 1, base + vec, 3 * base + 2 * vec + 1]):
            op = ["sum", "max", "avg", "min"][k % 4]
            gen = torch.Generator(device="cuda").manual_seed(500 + k)
            ins = [torch.randn(count, device="cuda", generator=gen).to(dtype) for _ in range(ranks)]
            raw = [torch.full((count + 16,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
            outs = [t[8:8 + count] for t in raw]
            comm.all_reduce(outs, ins, op=op)
            stack = torch.stack([t.float() for t in ins])
            ref = {"sum": stack.sum(0), "avg": stack.sum(0) / ranks, "max": stack.max(0).values, "min": stack.min(0).values}[op]
            for t, o in zip(raw, outs):
                assert (o.float() - ref).abs().max().item() <= tol, (count, op)
                assert (t[:8] == 7.0).all() and (t[8 + count:] == 7.0).all()
            part = ins[0].numel() // ranks + 1
            big = [torch.randn(part * ranks, device="cuda", generator=gen).to(dtype) for _ in range(ranks)]
            shard = [torch.empty(part, device="cuda", dtype=dtype) for _ in range(ranks)]
            comm.reduce_scatter(shard, big, op="max")
            most = torch.stack([t.float() for t in big]).max(0).values
            full = [torch.empty(part * ranks, device="cuda", dtype=dtype) for _ in range(ranks)]
            comm.all_gather(full, shard)
            for r in range(ranks):
                assert torch.equal(shard[r].float(), most[r * part:(r + 1) * part]) and torch.equal(full[r].float(), most)
        torch.cuda.synchronize()
        comm.check_async_error()
    finally:
        comm.close()
