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
            out, bits = {}, {}
            for parts in (1, 2, 4, 8):
                tcec.set_option("k_parts", parts)
                c = torch.full_like(c0, float("nan")) if beta == 0.0 else c0.clone()
                tcec.sgemm(a, b, c, alpha=alpha, beta=beta, policy=policy)
                tcec.device_status()
                out[parts] = (c.double() - exact).norm().item() / size
                bits[parts] = c
            # the option does divide: added in parts, some sums of a hundred and more round in another way
            if policy.endswith("_ec") and not policy.endswith("no_ec"):
                assert not any(torch.equal(bits[p], bits[q]) for p in bits for q in bits if p < q), (layouts, alpha)
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


def _undivided(call):
    tcec.set_option("k_parts", 1)
    out = call()
    tcec.set_option("k_parts", -1)
    return out


@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_ec", "fp16_no_ec"])
@pytest.mark.parametrize("m,n,k", [(900, 520, 3200), (300, 260, 5000)])
def test_host_operands_divide_as_one_device_call_does(m, n, k, policy):
    """Row panels have fewer tiles than the whole product, which alone decides."""
    gen = torch.Generator(device=DEV).manual_seed(8)
    a, b = _rand(gen, m, k), _rand(gen, k, n)
    want = tcec.sgemm(a, b, policy=policy)
    assert not torch.equal(want, _undivided(lambda: tcec.sgemm(a, b, policy=policy)))  # divided, that is
    ah, bh, ch = a.cpu().pin_memory(), b.cpu().pin_memory(), torch.empty((m, n)).pin_memory()
    for rows in (256, 512, 0):
        ch.fill_(float("nan"))
        tcec.sgemm_host(ah, bh, ch, policy=policy, panel_rows=rows)
        torch.cuda.current_stream().synchronize()
        assert torch.equal(ch, want.cpu()), rows
    tcec.device_status()


def test_a_batch_of_one_matrix_has_the_bits_of_a_larger_one():
    gen = torch.Generator(device=DEV).manual_seed(9)
    a, b = _rand(gen, 3, 200, 3000), _rand(gen, 3, 3000, 300)
    batch = tcec.sgemm_strided_batched(a, b)
    assert not torch.equal(batch[1], tcec.sgemm(a[1], b[1]))
    assert torch.equal(batch[1:2], tcec.sgemm_strided_batched(a[1:2], b[1:2]))
    c = [torch.zeros(200, 300, device=DEV)]
    tcec.sgemm_batched([a[1]], [b[1]], c)
    assert torch.equal(batch[1], c[0])
    assert torch.equal(batch[1], _undivided(lambda: tcec.sgemm(a[1], b[1])))


@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_ec", "fp16_no_ec"])
def test_undivided_calls_agree_at_long_k(policy):
    """What the options say of each other's bits, where K is long enough to be divided: forced kernels, a row range and a column
    range of packed operands, and the column-sharded calls."""
    gen = torch.Generator(device=DEV).manual_seed(10)
    m, n, k = 600, 520, 3000  # 25 tiles: four parts
    a, b = _rand(gen, m, k), _rand(gen, k, n)
    want = _undivided(lambda: tcec.sgemm(a, b, policy=policy))
    assert not torch.equal(want, tcec.sgemm(a, b, policy=policy))
    for name, values, default in (("cta_pair", (0, 1), -1), ("static_tiles", (1,), 0), ("narrow_tiles", (0, 32, 64, 128), -1),
                                  ("reserve_sms", (20,), 0), ("store_turn", (0,), 1), ("half_tiles", (0,), 1)):
        for value in values:
            tcec.set_option(name, value)
            try:
                got = tcec.sgemm(a, b, policy=policy) if name != "half_tiles" else _undivided(lambda: tcec.sgemm(a, b, policy=policy))
            finally:
                tcec.set_option(name, default)
            assert torch.equal(got, want), (name, value)
    ap, bp = tcec.pack_a(a, policy), tcec.pack_b(b, policy)
    oa, ob = tcec.packed_row_offset(512, k, policy), tcec.packed_row_offset(256, k, policy)
    part = _undivided(lambda: tcec.sgemm_packed(ap[oa:], bp[ob:], m - 512, n - 256, k, policy=policy))
    assert torch.equal(part, want[512:, 256:])
    shard = torch.empty(m, n, device=DEV)
    tcec.sgemm_column_shard(a, b, shard, m, k, policy=policy)
    assert torch.equal(shard, want)
    bh, ch = b.cpu().pin_memory(), torch.empty(m, n).pin_memory()
    tcec.sgemm_column_shard_host(a.cpu().pin_memory(), bh, ch, m, k, policy=policy, panel_rows=256)
    torch.cuda.current_stream().synchronize()
    assert torch.equal(ch, want.cpu())
    tcec.device_status()
