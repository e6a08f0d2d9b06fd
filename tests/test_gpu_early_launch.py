"""Calls that depend on one another, back to back on one stream: every kernel is set up beside the one before it and has to wait for
that one's results, whichever kernel it is.  The calls share four regions of memory, in which each writes what others read, read again
and write over; no other kernel and no synchronisation comes between.  The bits are those of the same calls with a synchronisation
after each."""
import random

import pytest
import torch

from wmma_extension_b200 import tcec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
FLOATS = 64 * 256 * 256  # of a region


class Machine:
    """Four regions and the calls on them; what a call needs besides (pointer tables, packed operands) is made beforehand."""

    def __init__(self, seed):
        gen = torch.Generator(device=DEV).manual_seed(seed)
        self.start = [torch.rand(FLOATS, generator=gen, device=DEV).mul_(2).sub_(1) for _ in range(4)]
        self.regions = [r.clone() for r in self.start]
        self.packed = [torch.empty(tcec.packed_bytes(700, 500), dtype=torch.uint8, device=DEV) for _ in range(2)]
        self.tables = {}

    def reset(self):
        for r, s in zip(self.regions, self.start):
            r.copy_(s)
        torch.cuda.synchronize()

    def view(self, region, *shape):
        count = 1
        for s in shape:
            count *= s
        return self.regions[region][:count].view(*shape)

    def single(self, n, m, k, a, b, c, policy="fp16_ec", beta=0.0):
        tcec.sgemm(self.view(a, m, k), self.view(b, k, n), self.view(c, m, n), alpha=k ** -0.5, beta=beta, policy=policy)

    def strided(self, batch, n, a, b, c, policy="fp16_ec", beta=0.0):
        x, y, z = (self.view(r, batch, n, n) for r in (a, b, c))
        tcec.sgemm_strided_batched(x, y, z, alpha=n ** -0.5, beta=beta, policy=policy)

    def table(self, batch, n, a, b, c):
        key = (batch, n, a, b, c)
        if key not in self.tables:
            self.tables[key] = [torch.tensor([self.regions[r].data_ptr() + 4 * n * n * i for i in range(batch)], device=DEV) for r in (a, b, c)]
        pa, pb, pc = self.tables[key]
        st = tcec.load().tcec_sgemm_batched(0, 0, 0, n, n, n, n ** -0.5, pa.data_ptr(), n, pb.data_ptr(), n, 0.0, pc.data_ptr(), n, batch, 0,
                                            torch.cuda.current_stream().cuda_stream)
        assert st == tcec.OK

    def complex(self, n, a, b, c, alpha=1.0):
        x, y, z = (torch.view_as_complex(self.view(r, n, n, 2)) for r in (a, b, c))
        tcec.cgemm(x, y, z, alpha=alpha / n ** 0.5)

    def pack(self, a, b, c):
        tcec.pack_a(self.view(a, 700, 500), "fp16_ec", self.packed[0])
        tcec.pack_b(self.view(b, 500, 300), "fp16_ec", self.packed[1])
        tcec.sgemm_packed(self.packed[0], self.packed[1], 700, 300, 500, self.view(c, 700, 300), alpha=500 ** -0.5)

    def scale(self, c):  # k = 0: an ordinary launch
        z = self.view(c, 600, 600)
        tcec.sgemm(z[:, :0], z[:0], z, beta=-1.0)


def calls(m):
    """name -> call(a, b, c) on regions"""
    return {
        "direct": lambda a, b, c: m.single(32, 32, 32, a, b, c),
        "direct, tf32, old values": lambda a, b, c: m.single(100, 90, 50, a, b, c, "tf32_ec", 0.5),
        "direct, 64 a matrix": lambda a, b, c: m.strided(1000, 64, a, b, c),
        "direct, 100 a matrix, old values": lambda a, b, c: m.strided(400, 100, a, b, c, "fp16_no_ec", -0.5),
        "FP32 tiles": lambda a, b, c: m.strided(64, 256, a, b, c),
        "FP32 tiles, old values": lambda a, b, c: m.strided(40, 256, a, b, c, "fp16_ec", 0.5),
        "FP32 tiles, by tables": lambda a, b, c: m.table(64, 256, a, b, c),
        "direct, by tables": lambda a, b, c: m.table(300, 48, a, b, c),
        "panels": lambda a, b, c: m.single(500, 300, 400, a, b, c),
        "panels, divided K, old values": lambda a, b, c: m.single(200, 300, 2000, a, b, c, "fp16_ec", 0.5),
        "panels, tf32": lambda a, b, c: m.single(1000, 1100, 1200, a, b, c, "tf32_ec"),
        "panels, pairs": lambda a, b, c: m.single(2000, 2000, 900, a, b, c, "fp16_no_ec"),
        "panels of a batch": lambda a, b, c: m.strided(3, 1000, a, b, c, "tf32_ec"),
        "packed": m.pack,
        "complex": lambda a, b, c: m.complex(300, a, b, c),
        "complex, complex alpha": lambda a, b, c: m.complex(200, a, b, c, 0.6 + 0.8j),
        "scaling": lambda a, b, c: m.scale(c),
    }


def run(machine, program, synchronise=False):
    table = calls(machine)
    for name, regions in program:
        table[name](*regions)
        if synchronise:
            torch.cuda.synchronize()


def check(machine, program):
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        machine.reset()
        run(machine, program, synchronise=True)
        want = [r.clone() for r in machine.regions]
        for _ in range(3):
            machine.reset()
            run(machine, program)
            torch.cuda.synchronize()
            for i, (got, w) in enumerate(zip(machine.regions, want)):
                assert torch.equal(got.view(torch.int32), w.view(torch.int32)), (i, program)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        run(machine, program)
    for _ in range(3):
        machine.reset()
        graph.replay()
        torch.cuda.synchronize()
        for i, (got, w) in enumerate(zip(machine.regions, want)):
            assert torch.equal(got.view(torch.int32), w.view(torch.int32)), (i, program)
    tcec.device_status()
    assert all(bool(torch.isfinite(w).all()) for w in want)


NAMES = ["direct", "direct, tf32, old values", "direct, 64 a matrix", "direct, 100 a matrix, old values", "FP32 tiles",
         "FP32 tiles, old values", "FP32 tiles, by tables", "direct, by tables", "panels", "panels, divided K, old values",
         "panels, tf32", "panels, pairs", "panels of a batch", "packed", "complex", "complex, complex alpha", "scaling"]


@pytest.mark.parametrize("first", NAMES)
def test_every_kernel_after_every_other(first):
    """The result of `first` is the other's operand, and the other writes over what `first` read."""
    machine = Machine(1)
    assert list(calls(machine)) == NAMES
    program = []
    for second in NAMES:
        program += [(first, (0, 1, 2)), (second, (2, 3, 0)), (first, (0, 3, 1)), (second, (1, 0, 3))]
        if len(program) >= 16:
            check(machine, program)
            program = []
    check(machine, program)


@pytest.mark.parametrize("seed", range(12))
def test_mixed_chains(seed):
    rng = random.Random(seed)
    machine = Machine(100 + seed)
    program = []
    for _ in range(24):
        name = rng.choice(NAMES)
        a, b, c = rng.sample(range(4), 3)
        if rng.random() < 0.2 and "old values" not in name and not name.startswith(("panels", "packed", "complex")):
            c = a  # in place
        program.append((name, (a, b, c)))
    check(machine, program)
