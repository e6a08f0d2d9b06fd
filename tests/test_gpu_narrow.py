"""The panel GEMM on narrow tiles against the wide kernels: the same bits at every width."""
import pytest
import torch

from wmma_extension_b200 import tcec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _default_options():
    yield
    for name, value in (("narrow_tiles", -1), ("direct_kernel", -1)):
        tcec.set_option(name, value)


@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_ec", "fp16_no_ec", "tf32_no_ec"])
@pytest.mark.parametrize("m,n,k", [
    (1, 1, 1), (7, 33, 31), (64, 520, 96), (72, 129, 33), (128, 128, 640), (129, 31, 65), (300, 257, 1000),
    (1000, 777, 333), (2100, 2000, 70),  # the last: several tiles per CTA at every width
])
def test_same_bits_at_every_width(m, n, k, policy):
    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    a = torch.rand((m, k), generator=gen, device=DEV).mul_(2).sub_(1)
    b = torch.rand((k, n), generator=gen, device=DEV).mul_(2).sub_(1)
    c0 = torch.rand((m, n + 3), generator=gen, device=DEV)
    tcec.set_option("direct_kernel", 0)
    for alpha, beta, col in ((1.0, 0.0, False), (-0.5, 0.75, False), (1.5, 0.25, True)):
        want = None
        for width in (0, 32, 64, 128):
            tcec.set_option("narrow_tiles", width)
            buf = c0.t().contiguous().t() if col else c0.clone()
            tcec.sgemm(a, b, buf[:, :n], alpha=alpha, beta=beta, policy=policy)
            tcec.device_status()
            if want is None:
                want = buf
            assert torch.equal(buf, want), (width, alpha, beta, col)


def test_packed_sub_range_at_every_width():
    """A sub-range that ends where its buffer does: the widths read row blocks one at a time, none beyond the operand."""
    gen = torch.Generator(device=DEV).manual_seed(9)
    m, n, k = 512, 768, 160
    a = torch.randn((m, k), generator=gen, device=DEV)
    b = torch.randn((k, n), generator=gen, device=DEV)
    ap, bp = tcec.pack_a(a), tcec.pack_b(b)
    want = tcec.sgemm(a, b)
    oa, ob = tcec.packed_row_offset(256, k), tcec.packed_row_offset(512, k)
    for width in (0, 32, 64, 128):
        tcec.set_option("narrow_tiles", width)
        assert torch.equal(tcec.sgemm_packed(ap[oa:], bp[ob:], 256, 256, k), want[256:, 512:]), width
    tcec.device_status()


def test_few_rows_by_packed_weights():
    """What the narrow tiles are chosen for: a handful of rows of A (only those are copied)."""
    gen = torch.Generator(device=DEV).manual_seed(10)
    for m in (1, 8, 9, 63, 65):
        a = torch.randn((m, 700), generator=gen, device=DEV)
        b = torch.randn((700, 1030), generator=gen, device=DEV)
        got = tcec.sgemm_packed(tcec.pack_a(a), tcec.pack_b(b), m, 1030, 700)
        exact = a.double() @ b.double()
        assert (got.double() - exact).norm() / exact.norm() < 1e-6
    tcec.device_status()
