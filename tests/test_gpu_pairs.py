"""The CTA-pair kernel where its launch is paced: the bits of the one-SM kernel, whatever else uses the pacing words."""
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


def test_paced_launches_overlap_on_streams_and_in_a_replayed_graph():
    """A graph replayed beside calls on the stream it was captured on shares that stream's word; a 64th stream has none."""
    a, b = _operands(5120, 4096, 5472, 7)
    want = _one_sm(a, b, "fp16_ec")
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(4)]
    outs = []
    for s in streams:
        with torch.cuda.stream(s):
            outs.append(tcec.sgemm(a, b))
    torch.cuda.synchronize()
    graph, captured = torch.cuda.CUDAGraph(), torch.zeros_like(want)
    with torch.cuda.graph(graph, stream=streams[0]):
        tcec.sgemm(a, b, captured)
    for _ in range(3):
        graph.replay()
        with torch.cuda.stream(streams[1]):
            outs.append(tcec.sgemm(a, b))
    torch.cuda.synchronize()
    assert torch.equal(captured, want) and all(torch.equal(o, want) for o in outs)
    tcec.device_status()
