"""Worker for the tests of the checking build of the library (B200CCL_LIBRARY=check is set by the
caller before this process starts). Every failure here is made on the host; no GPU faults.
socket-fault — a send proxy closes its socket after two slices: the ring kernels must leave their
               waits, the error must name the edge, and the communicator must refuse new work;
bounds       — the host is told to pass extents that are too short: the kernel must record the
               first bad index, skip those accesses and still run to its end;
separate-gpus — emulated ranks synchronise as ranks on GPUs of their own do: the ring's early credit and single
               group of warps at system scope, the peer kernels' barriers with their plan fingerprints;
separate-gpus-edges — the same at the edges: buffers that are misaligned alike and differently, batches of low-latency words
               with outputs of their own and in place;
canary       — the staging arena sits between two pages of canary bytes: they survive staged
               collectives, and a byte overwritten from the host is reported."""
import os
import sys

import torch

import nano_nccl_b200 as nn


def reference(ins, op):
    stack = torch.stack([t.float() for t in ins])
    return {"sum": stack.sum(0), "avg": stack.sum(0) / len(ins), "max": stack.max(0).values, "min": stack.min(0).values}[op]


def separate_gpus():
    """Every algorithm that a job on several GPUs may take, several calls in a row: lengths of one early-credit slice, of many
    slices and ragged ones for the ring; around the packs for the peer kernels; all three collectives."""
    cases = [("ring", t, c, r) for t, c in (("auto", 4), ("auto", 0), ("shm", 4)) for r in (2, 3, 8)]
    cases += [(a, "auto", 0, r) for a in ("oneshot", "twoshot", "ll") for r in (2, 3, 8)]
    for algo, transport, channels, ranks in cases:
        comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo=algo, transport=transport, channels=channels, wait_timeout_ms=3000)
        assert "as on GPUs of their own" in comm.describe()
        for dtype, tol in ((torch.float32, 1e-5), (torch.bfloat16, 2e-1)):  # bf16: the ring rounds once per hop, sums to 30
            counts = [1024, 4096, 16384, 2048, 4096, 1024, 8192] * 3 + ([1 << 15, 6] if algo == "ll" else [(1 << 20) + 8, 300001, 7])
            for i, count in enumerate(counts):
                op = ["sum", "avg", "max", "min"][i % 4]
                gen = torch.Generator(device="cuda").manual_seed(900 + i)
                ins = [torch.randn(count, device="cuda", generator=gen).to(dtype) for _ in range(ranks)]
                outs = [torch.full_like(t, float("nan")) for t in ins]
                comm.all_reduce(outs, ins, op=op)
                assert comm.last_call()["algo"] == algo
                for o in outs:
                    assert (o.float() - reference(ins, op)).abs().max().item() <= tol, (algo, transport, ranks, count, op)
            for block in () if algo == "ll" else (2048, 1 << 17, 1001, 3):
                ins = [torch.randn(block * ranks, device="cuda").to(dtype) for _ in range(ranks)]
                shards = [torch.empty(block, device="cuda", dtype=dtype) for _ in range(ranks)]
                full = [torch.empty(block * ranks, device="cuda", dtype=dtype) for _ in range(ranks)]
                comm.reduce_scatter(shards, ins, op="max")
                comm.all_gather(full, shards)
                most = reference(ins, "max").to(dtype)
                assert all(torch.equal(f, most) for f in full), (algo, transport, ranks, block)
        torch.cuda.synchronize()
        comm.check_async_error()
        comm.close()


def separate_gpus_edges():
    """The peer kernels with their meetings over flags: the elements before the first pack and behind the last one of views that
    are misaligned alike, for every width of pack; the low-latency exchange between threads of different CTAs on both sides of
    every size of batch. Max and min are exact; sums are added in rank order in fp32 and rounded once."""
    def combined(ins, op):
        acc = ins[0].float()
        for t in ins[1:]:
            acc = acc + t.float() if op in ("sum", "avg") else (torch.maximum if op == "max" else torch.minimum)(acc, t.float())
        return (acc * torch.tensor(1.0, device="cuda").div(len(ins)) if op == "avg" else acc).to(ins[0].dtype)

    gen = torch.Generator(device="cuda").manual_seed(77)
    for algo in ("oneshot", "twoshot"):
        for ranks in (2, 3, 8):
            comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo=algo, wait_timeout_ms=3000)
            assert "as on GPUs of their own" in comm.describe()
            for dtype in (torch.float32, torch.bfloat16):
                esz = torch.empty(0, dtype=dtype).element_size()
                for k, count in enumerate([1, 32 // esz, 48 // esz - 1, 62 // esz, 64 // esz + 1, 257, 30001, (1 << 18) + 5]):
                    for shifts in ([1] * ranks, [5] * ranks, [16 // esz + 1] * ranks, [32 // esz - 1] * ranks, [(3 * r) % 5 for r in range(ranks)]):
                        op = ["sum", "avg", "max", "min"][(k + shifts[0]) % 4]
                        ins = [torch.randn(count + 64, device="cuda", generator=gen).to(dtype)[s:s + count] for s in shifts]
                        raw = [torch.full((count + 64,), 7.0, device="cuda", dtype=dtype) for _ in range(ranks)]
                        outs = [t[s:s + count] for t, s in zip(raw, shifts)]
                        expect = combined(ins, op)
                        if algo == "twoshot" and k % 2:  # in place
                            for t, o in zip(ins, outs):
                                o.copy_(t)
                            comm.all_reduce(outs, outs, op=op)
                        else:
                            comm.all_reduce(outs, ins, op=op)
                        assert comm.last_call()["algo"] == algo
                        for t, o, s in zip(raw, outs, shifts):
                            assert torch.equal(o, expect), (algo, ranks, dtype, count, shifts, op)
                            assert (t[:s] == 7.0).all() and (t[s + count:] == 7.0).all(), (algo, ranks, dtype, count, shifts, op)
            comm.check_async_error()
            comm.close()
    for ranks in (2, 3, 8):
        comm = nn.Communicator(devices=[0], loopback_ranks=ranks, algo="ll", wait_timeout_ms=3000)
        for k, words in enumerate([4096, 4097, 5, 16384, 16385, 32768, 1, 32767, 20480, 16383] * 2):
            ins = [torch.randn(words * 2, device="cuda", generator=gen).half() for _ in range(ranks)]
            outs = [torch.full_like(t, float("nan")) for t in ins]
            op = ["sum", "avg", "max", "min"][k % 4]
            expect = combined(ins, op)
            comm.all_reduce(outs, ins, op=op)
            assert comm.last_call()["algo"] == "ll" and all(torch.equal(o, expect) for o in outs), (ranks, words, op)
            comm.all_reduce(ins, ins, op=op)
            assert all(torch.equal(o, expect) for o in ins), (ranks, words, op, "in place")
        comm.check_async_error()
        comm.close()


def main():
    mode = sys.argv[1]
    torch.cuda.set_device(0)
    assert os.environ.get("B200CCL_LIBRARY") == "check"
    if mode == "socket-fault":
        comm = nn.Communicator(devices=[0], loopback_ranks=2, transport="socket", channels=2, wait_timeout_ms=3000)
        numel = 8 << 20  # 32 MiB per rank: many slices per channel
        ins = [torch.randn(numel, device="cuda") for _ in range(2)]
        outs = [torch.zeros_like(t) for t in ins]
        comm.all_reduce(outs, ins)
        torch.cuda.synchronize()  # returns: the proxy's error raised the abort word, the kernels left their waits
        try:
            comm.check_async_error()
            raise SystemExit("expected the injected socket failure")
        except nn.B200CclError as e:
            text = str(e)
            assert "socket" in text and "injected" in text, text
            for part in ("source=", "destination=", "channel=", "step="):
                assert part in text, text
            print("detected:", text)
        try:
            comm.all_reduce(outs, ins)
            raise SystemExit("a failed communicator must refuse new work")
        except nn.B200CclError:
            pass
        assert torch.ones(8, device="cuda").sum().item() == 8  # the context is still usable
        comm.close()
    elif mode == "bounds":
        comm = nn.Communicator(devices=[0], loopback_ranks=4, algo="twoshot", wait_timeout_ms=3000)
        numel = 1 << 16
        ins = [torch.randn(numel, device="cuda") for _ in range(4)]
        outs = [torch.full_like(t, -7.0) for t in ins]
        comm.all_reduce(outs, ins)
        torch.cuda.synchronize()
        try:
            comm.check_async_error()
            raise SystemExit("expected the self-check to fire")
        except nn.B200CclError as e:
            assert "self-check" in str(e) and "beyond the buffer extent" in str(e), str(e)
            print("detected:", e)
        # packs beyond the (shrunk) extent were skipped, everything below it was reduced
        ref = torch.stack(ins).sum(0)
        shrink_elems = int(os.environ["B200CCL_DEBUG_SHRINK_EXTENT"]) * comm.last_call()["pack_bytes"] // 4
        good = numel - shrink_elems
        for o in outs:
            assert (o[:good] - ref[:good]).abs().max().item() <= 1e-5
            assert (o[good:] == -7.0).all()
        comm.close()
    elif mode == "separate-gpus":
        separate_gpus()
    elif mode == "separate-gpus-edges":
        separate_gpus_edges()
    elif mode == "canary":
        smash = os.environ.pop("B200CCL_DEBUG_SMASH_CANARY", None)
        comm = nn.Communicator(devices=[0], loopback_ranks=4, algo="pipeline", wait_timeout_ms=3000, staging_bytes=8 << 20)
        for numel in (1 << 20, (3 << 20) + 4, 4096):
            ins = [torch.randn(numel, device="cuda") for _ in range(4)]
            outs = [torch.empty_like(t) for t in ins]
            comm.all_reduce(outs, ins)
            torch.cuda.synchronize()
            comm.check_async_error()   # includes the canary check in this build
            ref = torch.stack(ins).sum(0)
            assert all((o - ref).abs().max().item() <= 1e-5 for o in outs)
        if smash:
            os.environ["B200CCL_DEBUG_SMASH_CANARY"] = "1"
            try:
                comm.check_async_error()
                raise SystemExit("expected the canary check to fire")
            except nn.B200CclError as e:
                assert "canary overwritten" in str(e) and "after the arena" in str(e), str(e)
                print("detected:", e)
        comm.close()
    print("WORKER OK")


if __name__ == "__main__":
    main()
