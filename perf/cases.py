"""What the speed of this library is measured on: collective calls through the Python communicator
on one GPU, alone (one rank) or with 2 to 8 ranks that share the device.

A case is a plain dict:

  collective  all_reduce | reduce_scatter | all_gather
  ranks       1 to 8; more than one means ``Communicator(devices=[0], loopback_ranks=ranks)``
  dtype       float | fp16 | bf16
  op          sum | avg | max | min (all_gather: sum, unused)
  count       elements of the smaller side of one rank: the message of an all_reduce, the block of a
              reduce_scatter (its input is ranks * count) or of an all_gather (its output is)
  algo        auto | twoshot | oneshot | ll | ring, as the constructor takes it
  transport   auto | shm, likewise
  in_place    all_reduce only: reduce the tensors into themselves
  symmetric   buffers from ``Communicator.empty`` instead of ordinary tensors
  shift       elements by which every buffer starts past its (aligned) allocation: views such as x[1:]
"""
import math

import torch

from nano_nccl_b200 import Communicator

DTYPES = {"float": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
BYTES = {"float": 4, "fp16": 2, "bf16": 2}
LARGEST = 2 << 30  # bytes of all ranks' messages together, at most


def _case(name, collective, ranks, dtype, op, count, algo="auto", transport="auto", in_place=False, symmetric=False, shift=0):
    c = {"collective": collective, "ranks": ranks, "dtype": dtype, "op": op, "count": count, "algo": algo,
         "transport": transport, "in_place": in_place, "symmetric": symmetric, "shift": shift}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # A small message of a job that runs on one GPU only: the call itself is the cost.
        _case("one_rank_8KiB", "all_reduce", 1, "bf16", "sum", 4096),
        # bench.py's default workload at one GPU.
        _case("one_rank_64MiB", "all_reduce", 1, "float", "sum", 16 << 20),
        # Latency: a metric or a loss that every rank contributes a few values to.
        _case("sum8_4KiB", "all_reduce", 8, "float", "sum", 1024),
        # The kernel of nodes without multicast, asked for by name, as it is profiled on one GPU.
        _case("twoshot4_8MiB", "all_reduce", 4, "bf16", "sum", 4 << 20, algo="twoshot"),
        # A length that is no multiple of anything.
        _case("max4_odd", "all_reduce", 4, "fp16", "max", 1000003),
        # A gradient bucket: the default bucket size of BucketAllReducer, averaged in place in symmetric memory.
        _case("bucket8_25MiB", "all_reduce", 8, "bf16", "avg", (25 << 20) // 2, in_place=True, symmetric=True),
        # The headline size: 64 MiB of float32 per rank.
        _case("sum8_64MiB", "all_reduce", 8, "float", "sum", 16 << 20),
        # The largest message of the benchmark's sweep.
        _case("sum2_1GiB", "all_reduce", 2, "float", "sum", 256 << 20),
        # Sharded data parallelism: gradients are reduce-scattered, parameters are gathered.
        _case("scatter8_4MiB", "reduce_scatter", 8, "bf16", "avg", 2 << 20),
        _case("gather8_4MiB", "all_gather", 8, "bf16", "sum", 2 << 20),
        # The ring with Simple FIFOs over device memory, and over host memory for GPUs that cannot address each other.
        _case("ring4_16MiB", "all_reduce", 4, "float", "sum", 4 << 20, algo="ring"),
        _case("shm4_4MiB", "all_reduce", 4, "float", "sum", 1 << 20, transport="shm"),
    ]


def draw(rng):
    """1 to 8 ranks, every collective, type and operator, 1 KiB to 1 GiB per rank, half of the lengths ragged."""
    dtype = rng.choice(["float", "fp16", "bf16"])
    collective = rng.choice(["all_reduce"] * 4 + ["reduce_scatter", "all_gather"])
    ranks = rng.choice([1, 2, 3, 4, 5, 6, 7, 8, 8, 4])
    algo, transport = "auto", "auto"
    if ranks > 1:
        special = rng.random()
        if special < 0.08:
            algo = "ring"
        elif special < 0.12:
            transport = "shm"
        elif special < 0.28 and collective == "all_reduce":
            algo = rng.choice(["twoshot", "oneshot", "ll"])
    # The message that one rank holds (the longer side of a reduce_scatter or an all_gather).
    most = min(1 << 30, LARGEST // ranks)
    if algo == "ll":
        most = 128 << 10
    elif algo == "oneshot":
        most = 4 << 20
    elif algo == "ring":
        most = 64 << 20
    elif transport == "shm":
        most = 8 << 20
    message = int(math.exp(rng.uniform(math.log(1024), math.log(most))))
    count = max(1, message // BYTES[dtype] // (1 if collective == "all_reduce" else ranks))
    if algo == "ll":
        count = max(2, count // 2 * 2)  # whole 4-byte words are all that it takes
    elif rng.random() < 0.5:
        count = max(64, count // 64 * 64)
    shift = 1 if algo != "ll" and rng.random() < 0.08 else 0
    op = "sum" if collective == "all_gather" else rng.choice(["sum", "sum", "avg", "max", "min"])
    # A sum that is repeated in place would grow without bound: averages and extremes stay where they are.
    in_place = collective == "all_reduce" and ranks > 1 and op != "sum" and algo != "oneshot" and rng.random() < 0.3
    symmetric = shift == 0 and transport == "auto" and rng.random() < 0.25
    return _case("", collective, ranks, dtype, op, count, algo, transport, in_place, symmetric, shift)


class State:
    """The communicator that a job keeps, one input and one output tensor per rank, and the call to make."""

    def __init__(self, comm, collective, op, ins, outs):
        self.comm, self.collective, self.op, self.ins, self.outs = comm, collective, op, ins, outs


_communicators = {}


def _communicator(case, own):
    """A job creates its communicator once. One that gives out symmetric memory belongs to a single state, so
    that the memory goes when the state does."""
    key = (case["ranks"], case["algo"], case["transport"])
    if not own and key in _communicators:
        return _communicators[key]
    torch.cuda.set_device(0)
    comm = Communicator(devices=[0], loopback_ranks=case["ranks"] if case["ranks"] > 1 else 0, algo=case["algo"],
                        transport=case["transport"])
    if not own:
        _communicators[key] = comm
    return comm


def _lengths(case):
    n, count = case["ranks"], case["count"]
    return (count * n if case["collective"] == "reduce_scatter" else count,
            count * n if case["collective"] == "all_gather" else count)


def prepare(case, seed):
    n, dtype, shift = case["ranks"], DTYPES[case["dtype"]], case["shift"]
    in_len, out_len = _lengths(case)
    comm = _communicator(case, case["symmetric"])

    def buffers(length):
        if case["symmetric"]:
            got = comm.empty(length, dtype)
            return got if isinstance(got, list) else [got]
        return [torch.empty(length + shift, dtype=dtype, device="cuda")[shift:] for _ in range(n)]

    ins = buffers(in_len)
    outs = ins if case["in_place"] else buffers(out_len)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for t in ins:  # gradients and activations: centred, most of them small
        t.normal_(0.0, 1.0, generator=gen)
    return State(comm, case["collective"], case["op"], ins if n > 1 else ins[0], outs if n > 1 else outs[0])


def run(state):
    if state.collective == "all_reduce":
        return state.comm.all_reduce(state.outs, state.ins, op=state.op)
    if state.collective == "reduce_scatter":
        return state.comm.reduce_scatter(state.outs, state.ins, op=state.op)
    return state.comm.all_gather(state.outs, state.ins)


def work(case):
    """Every rank's input is read once and every rank's output is written once; a reduction combines all ranks' elements."""
    n = case["ranks"]
    in_len, out_len = _lengths(case)
    reduced = 0 if case["collective"] == "all_gather" else (n - 1) * in_len
    return {"bytes": n * (in_len + out_len) * BYTES[case["dtype"]], "flops": reduced}


def tolerance(case):
    """Copies and extremes are exact. Sums are added in float32 in any order and rounded to the type once, or, in
    the ring, once per hop."""
    if case["ranks"] == 1 or case["collective"] == "all_gather" or case["op"] in ("max", "min"):
        return "exact"
    return {"rel": {"float": 1e-6, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
