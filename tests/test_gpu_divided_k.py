"""Panel products whose K is divided among the CTAs of a cluster: against FP64 beside the undivided kernel, over every number of
parts, edge and store path."""
import pytest
import torch

from wmma_extension_b200 import tcec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _default_options():
    yield
    tcec.set_option("k_parts", -1)


def _rand(gen, *shape):
    return torch.rand(shape, generator=gen, device=DEV).mul_(2).sub_(1)


def _error(got, exact):
    return ((got.double() - exact).norm() / exact.norm()).item()


@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_ec", "fp16_no_ec", "tf32_no_ec"])
@pytest.mark.parametrize("m,n,k", [
    (1, 129, 1200), (64, 500, 4096), (129, 1, 1233), (129, 257, 2000), (100, 1000, 1801), (300, 130, 5000), (7, 130, 257),
])
def test_divided_k_is_no_further_from_fp64_than_undivided(m, n, k, policy):
    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    for layouts in ("rrr", "rcc", "crr", "ccc"):
        a, b, c0 = ((_rand(gen, r, c) if l == "r" else _rand(gen, c, r).t()) for l, r, c in
                    zip(layouts, (m, k, m), (k, n, n)))
        for alpha, beta in ((1.0, 0.0), (1.5, -0.5)):
            exact = alpha * (a.double() @ b.double()) + beta * c0.double()
            # Errors relative to what the elements of C are expected to be (products of elements of variance 1/3), not to what they
            # are: a single element may lie close to zero.
            size = abs(alpha) * (m * n * k) ** 0.5 / 3
            out = {}
            for parts in (1, 2, 4, 8):
                tcec.set_option("k_parts", parts)
                c = torch.full_like(c0, float("nan")) if beta == 0.0 else c0.clone()
                tcec.sgemm(a, b, c, alpha=alpha, beta=beta, policy=policy)
                tcec.device_status()
                out[parts] = (c.double() - exact).norm().item() / size
            # On few elements the undivided error may be small by chance.  Adding the parts rounds once per part, by at most 2^-24
            # of sums that are seldom larger than three times the expected size.
            for parts in (2, 4, 8):
                assert out[parts] <= 1.05 * out[1] + 3 * parts * 2.0 ** -24 / (m * n) ** 0.5, (layouts, alpha, parts, out)


def test_a_call_alone_divides_and_few_rows_stay_in_their_matrix():
    """64 x 4096 x 4096 on packed operands: the automatic choice divides; rows and columns around C stay as they are."""
    gen = torch.Generator(device=DEV).manual_seed(2)
    a, b = _rand(gen, 64, 4096), _rand(gen, 4096, 4096)
    exact = a.double() @ b.double()
    ap, bp = tcec.pack_a(a), tcec.pack_b(b)
    buf = torch.full((66, 4104), 3.0, device=DEV)
    tcec.sgemm_packed(ap, bp, 64, 4096, 4096, buf[1:65, 4:4100])
    tcec.device_status()
    assert _error(buf[1:65, 4:4100], exact) < 3e-7
    buf[1:65, 4:4100] = 3.0
    assert bool((buf == 3.0).all())
    auto = tcec.sgemm_packed(ap, bp, 64, 4096, 4096)
    tcec.set_option("k_parts", 1)
    whole = tcec.sgemm_packed(ap, bp, 64, 4096, 4096)
    # largest error of either 6e-6 of the root mean square, 64 / 3
    assert not torch.equal(auto, whole) and torch.allclose(auto, whole, rtol=0, atol=2 * 6e-6 * 64 / 3)


def test_a_captured_call_divides_alike():
    gen = torch.Generator(device=DEV).manual_seed(5)
    a, b = _rand(gen, 330, 2500), _rand(gen, 2500, 129)
    want = tcec.sgemm(a, b)
    side, graph, captured = torch.cuda.Stream(), torch.cuda.CUDAGraph(), torch.zeros_like(want)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        tcec.sgemm(a, b)
    side.synchronize()
    with torch.cuda.graph(graph, stream=side):
        tcec.sgemm(a, b, captured)
    for _ in range(3):
        captured.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, want)
    tcec.device_status()


@pytest.mark.parametrize("batch,m,n", [(1, 128, 128), (3, 256, 200)])
def test_calls_with_another_kernel_under_capture_stay_undivided(batch, m, n):
    gen = torch.Generator(device=DEV).manual_seed(6)
    a, b = _rand(gen, batch, m, 3000), _rand(gen, batch, 3000, n)
    auto = tcec.sgemm_strided_batched(a, b)
    tcec.set_option("k_parts", 1)
    assert torch.equal(auto, tcec.sgemm_strided_batched(a, b))


def test_non_finite_operands_stay_in_their_rows_and_columns():
    gen = torch.Generator(device=DEV).manual_seed(3)
    a, b = torch.randn((40, 3000), generator=gen, device=DEV), torch.randn((3000, 200), generator=gen, device=DEV)
    a[3, 2999] = float("nan")
    b[7, 150] = float("inf")
    bad = ~torch.isfinite(tcec.sgemm(a, b, policy="tf32_ec"))
    want = torch.zeros_like(bad)
    want[3, :] = True
    want[:, 150] = True
    assert torch.equal(bad, want)
