"""The CTA-pair kernel where its launch is paced or draws its tiles: the bits of the one-SM kernel, whatever else runs."""
import ctypes
import time

import pytest
import torch

from wmma_extension_b200 import tcec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _default_options():
    yield
    tcec.set_option("cta_pair", -1)


def _operands(m, n, k, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.rand(m, k, generator=gen, device=DEV).mul_(2).sub_(1), torch.rand(k, n, generator=gen, device=DEV).mul_(2).sub_(1))


def _one_sm(a, b, policy):
    tcec.set_option("cta_pair", 0)
    want = tcec.sgemm(a, b, policy=policy)
    tcec.set_option("cta_pair", -1)
    return want


# four rounds of tiles and more on 74 pairs, panels of a wave just above 100 MB; ragged sizes; K that is no multiple of what a count covers
@pytest.mark.parametrize("m,n,k,policy", [
    (5120, 4096, 5472, "fp16_ec"), (5000, 4090, 5999, "fp16_ec"), (9000, 2390, 5541, "fp16_ec"), (5120, 4096, 2800, "tf32_ec"),
    (5120, 4096, 11000, "fp16_no_ec"),
])
def test_paced_pairs_have_the_bits_of_single_sms(m, n, k, policy):
    a, b = _operands(m, n, k, m + k)
    got = [tcec.sgemm(a, b, policy=policy) for _ in range(2)]
    tcec.device_status()
    want = _one_sm(a, b, policy)
    assert torch.equal(got[0], want) and torch.equal(got[1], want)


# long enough to draw tiles, paced or not: K of one, two and 43 K blocks, tiles that are cut on both sides, one tile row, a round and a bit
@pytest.mark.parametrize("m,n,k,policy", [
    (40000, 50000, 64, "fp16_ec"), (45000, 45001, 64, "tf32_ec"), (60001, 70001, 31, "fp16_ec"), (10000, 9500, 1350, "fp16_ec"),
    (256, 40000, 12500, "fp16_ec"), (2500, 2100, 24000, "fp16_ec"), (2500, 2100, 24000, "tf32_ec"),
])
def test_drawn_tiles_have_the_bits_of_single_sms(m, n, k, policy):
    a, b = _operands(m, n, k, m + k)
    got = [tcec.sgemm(a, b, policy=policy) for _ in range(2)]
    tcec.device_status()
    want = _one_sm(a, b, policy)
    assert torch.equal(got[0], want) and torch.equal(got[1], want)
    tcec.set_option("static_tiles", 1)
    tcec.set_option("cta_pair", 1)
    try:
        assert torch.equal(tcec.sgemm(a, b, policy=policy), want)
    finally:
        tcec.set_option("static_tiles", 0)


@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_ec"])
def test_a_long_call_waits_for_no_sms_that_another_kernel_holds(policy):
    """Four CTAs of another stream's product hold four SMs for longer than the call takes.  The pairs that have none of them do it all
    (70 of 74: 1.06 times as long); with a share of its own for every pair it took 1.61 to 1.88 times as long."""
    held = torch.rand(128, 1 << 20, device=DEV)
    a, b = _operands(8192, 8192, 4096, 3)
    c = torch.empty(8192, 8192, device=DEV)
    side = torch.cuda.Stream()

    def timed():
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        start.record()
        tcec.sgemm(a, b, c, policy=policy)
        end.record()
        return start, end

    def hold():
        tcec.set_option("direct_kernel", 1)  # one CTA a matrix
        try:
            with torch.cuda.stream(side):
                tcec.sgemm_strided_batched(held.expand(4, 128, 1 << 20), held.t().expand(4, 1 << 20, 128))
        finally:
            tcec.set_option("direct_kernel", -1)
        event = torch.cuda.Event()
        event.record(side)
        return event

    hold()
    for _ in range(3):
        timed()
    torch.cuda.synchronize()
    alone, beside = [], []
    for _ in range(5):
        start, end = timed()
        end.synchronize()
        alone.append(start.elapsed_time(end))
    want = c.clone()
    for _ in range(5):
        c.fill_(float("nan"))
        torch.cuda.synchronize()
        holder = hold()
        time.sleep(0.003)
        start, end = timed()
        end.synchronize()
        assert not holder.query()  # it was there all the while
        torch.cuda.synchronize()
        beside.append(start.elapsed_time(end))
        assert torch.equal(c, want)
    tcec.device_status()
    assert sorted(beside)[2] < 1.35 * sorted(alone)[2], (alone, beside)


def test_paced_launches_overlap_on_streams_and_in_a_replayed_graph():
    """Products of packed operands, which share nothing else.  A graph replayed beside calls on the stream that it was captured on shares
    that stream's pacing words."""
    m, n, k = 5120, 4096, 5472
    a, b = _operands(m, n, k, 7)
    want = _one_sm(a, b, "fp16_ec")
    ap, bp = tcec.pack_a(a), tcec.pack_b(b)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(4)]
    outs = [torch.zeros_like(want) for _ in range(16)]
    captured = torch.zeros_like(want)
    torch.cuda.synchronize()
    for s, out in zip(streams, outs):
        with torch.cuda.stream(s):
            tcec.sgemm_packed(ap, bp, m, n, k, out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        tcec.sgemm_packed(ap, bp, m, n, k, captured)
    for i in range(3):
        captured.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[1]):
            for _ in range(4):
                graph.replay()
        with torch.cuda.stream(streams[0]):
            for j in range(4):
                tcec.sgemm_packed(ap, bp, m, n, k, outs[4 + 4 * i + j])
        torch.cuda.synchronize()
        assert torch.equal(captured, want)
    assert all(torch.equal(o, want) for o in outs)
    tcec.device_status()


def test_more_streams_than_there_are_lines():
    """Every stream beyond the 63rd draws its tiles from counters of its own and is not paced."""
    cudart = torch.cuda.cudart()
    handles = []
    for _ in range(70):  # torch's own streams are fewer
        handle = ctypes.c_void_p(0)
        assert int(cudart.cudaStreamCreate(ctypes.addressof(handle))) == 0
        handles.append(handle.value)
    try:
        for m, n, k in ((5120, 4096, 5472), (4900, 5000, 5300)):  # paced; paced and drawn
            a, b = _operands(m, n, k, 8)
            want = _one_sm(a, b, "fp16_ec")
            ap, bp = tcec.pack_a(a), tcec.pack_b(b)
            outs = [torch.zeros_like(want) for _ in handles]
            torch.cuda.synchronize()
            for _ in range(2):
                for h, out in zip(handles, outs):
                    with torch.cuda.stream(torch.cuda.ExternalStream(h)):
                        tcec.sgemm_packed(ap, bp, m, n, k, out)
            torch.cuda.synchronize()
            assert all(torch.equal(o, want) for o in outs)
            del outs
        tcec.device_status()
    finally:
        torch.cuda.synchronize()
        tcec.destroy()  # the lines are free again
        for h in handles:
            cudart.cudaStreamDestroy(h)
