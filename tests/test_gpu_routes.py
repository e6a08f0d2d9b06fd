"""Calls whose kernel is chosen from their sizes: the same bits on either side of a choice, and no workspace where none can be
allocated."""
import pytest
import torch

from wmma_extension_b200 import tcec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _default_options():
    yield
    tcec.set_option("path", 0)


def _rand(gen, *shape):
    return torch.rand(shape, generator=gen, device=DEV).mul_(2).sub_(1)


@pytest.mark.parametrize("batch,m,n,k", [
    (2, 256, 256, 512), (2, 1024, 516, 1028),  # few tiles: from panels
    (90, 256, 132, 96), (40, 300, 260, 1028),  # many: on the FP32-tile kernel
])
def test_strided_batches_have_the_bits_of_the_panel_path(batch, m, n, k):
    gen = torch.Generator(device=DEV).manual_seed(batch + m)
    a, b, c0 = _rand(gen, batch, m, k), _rand(gen, batch, k, n), _rand(gen, batch, n, m)
    for transposed, alpha, beta in ((False, 1.0, 0.0), (True, -0.5, 0.75)):
        out = []
        for path in (1, 0):
            tcec.set_option("path", path)
            c = c0.clone()
            tcec.sgemm_strided_batched(a, b, c.transpose(1, 2) if transposed else c.view(batch, m, n), alpha=alpha, beta=beta)
            tcec.device_status()
            out.append(c)
        assert torch.equal(out[0], out[1]), (transposed, alpha, beta)


@pytest.mark.parametrize("batch,m,n,k", [(2, 256, 256, 512), (1, 100, 128, 700), (3, 128, 40, 3000)])
def test_a_first_call_may_be_captured(batch, m, n, k):
    """On a stream that has no workspace yet such a call, which would otherwise run from panels, takes the kernel without one."""
    gen = torch.Generator(device=DEV).manual_seed(k)
    a, b = _rand(gen, batch, m, k), _rand(gen, batch, k, n)
    torch.cuda.synchronize()
    tcec.destroy()  # no stream has a workspace
    want = tcec.sgemm_strided_batched(a, b)  # the library's state exists again, and this stream's workspace
    c = torch.zeros_like(want)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        tcec.sgemm_strided_batched(a, b, c)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(c, want)
    tcec.device_status()


@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_ec"])
@pytest.mark.parametrize("batch,m,n,k", [(1, 128, 128, 192), (1, 128, 128, 193), (1, 33, 128, 1030), (30, 100, 64, 500), (120, 20, 40, 700)])
def test_small_matrices_have_the_bits_of_the_panel_path(batch, m, n, k, policy):
    gen = torch.Generator(device=DEV).manual_seed(batch + k)
    a, b = _rand(gen, batch, m, k), _rand(gen, batch, k, n)
    out = []
    for path in (1, 0):
        tcec.set_option("path", path)
        out.append(tcec.sgemm_strided_batched(a, b, policy=policy))
        tcec.device_status()
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("batch,mn", [(40, 300), (90, 256), (100, 64), (3, 100)])
def test_results_over_their_operands(batch, mn):
    """In place, and one matrix on (C_i over A_i+1): as if the operands had been read before anything is written."""
    gen = torch.Generator(device=DEV).manual_seed(mn)
    pool, w = _rand(gen, batch + 1, mn, mn), _rand(gen, batch, mn, mn)
    want = tcec.sgemm_strided_batched(pool[:batch].clone(), w)
    for shift in (0, 1):
        x = pool.clone()
        tcec.sgemm_strided_batched(x[:batch], w, x[shift:shift + batch])
        assert torch.equal(x[shift:shift + batch], want), shift
    x = pool.clone()
    tcec.sgemm_batched(list(x[:batch]), list(w), list(x[:batch]))
    assert torch.equal(x[:batch], want)
    # B in place, C column-major
    want_t = tcec.sgemm_strided_batched(w, pool[:batch].transpose(1, 2).clone())
    x = pool[:batch].clone()
    tcec.sgemm_strided_batched(w, x.transpose(1, 2), x.transpose(1, 2))
    assert torch.equal(x.transpose(1, 2), want_t)
    tcec.device_status()


def test_a_single_product_in_place():
    gen = torch.Generator(device=DEV).manual_seed(8)
    for mn in (100, 700):
        a, w = _rand(gen, mn, mn), _rand(gen, mn, mn)
        want = tcec.sgemm(a, w)
        assert torch.equal(tcec.sgemm(a, w, a), want)
    tcec.device_status()


def test_tables_captured_behind_a_strided_call():
    """A strided call of the shape has sized the stream's workspace: the call by tables is then launches only."""
    gen = torch.Generator(device=DEV).manual_seed(11)
    batch, m, n, k = 120, 160, 160, 1024
    a, b = _rand(gen, batch, m, k), _rand(gen, batch, k, n)
    torch.cuda.synchronize()
    tcec.destroy()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        tcec.set_option("path", 1)
        want = tcec.sgemm_strided_batched(a, b)
        tcec.set_option("path", 0)
    s.synchronize()
    c = torch.zeros_like(want)
    tables = [torch.tensor([x.data_ptr() for x in t], dtype=torch.int64, device=DEV) for t in (a, b, c)]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        st = tcec.load().tcec_sgemm_batched(0, 0, 0, m, n, k, 1.0, tables[0].data_ptr(), k, tables[1].data_ptr(), n, 0.0,
                                            tables[2].data_ptr(), n, batch, 0, torch.cuda.current_stream().cuda_stream)
    assert st == tcec.OK
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(c, want)
    tcec.device_status()
