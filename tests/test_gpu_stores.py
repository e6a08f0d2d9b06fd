"""How C leaves the panel kernels: every path of the stores (whole and ragged blocks, aligned rows or not, either order, with
and without old values) against the product, bit for bit; nothing outside the matrix is written."""
import pytest
import torch

from wmma_extension_b200 import tcec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
KERNELS = {"narrow 32": {"narrow_tiles": 32}, "narrow 64": {"narrow_tiles": 64}, "narrow 128": {"narrow_tiles": 128},
           "one SM": {"cta_pair": 0, "narrow_tiles": 0}, "pair": {"cta_pair": 1, "narrow_tiles": 0}}
DEFAULTS = {"narrow_tiles": -1, "cta_pair": -1, "path": 0, "half_tiles": 1}


@pytest.fixture(autouse=True)
def _default_options():
    yield
    for name, value in DEFAULTS.items():
        tcec.set_option(name, value)


@pytest.mark.parametrize("kernel", list(KERNELS))
@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_no_ec"])
def test_every_way_to_store(kernel, policy):
    gen = torch.Generator(device=DEV).manual_seed(12)
    k = 40
    for name, value in dict(KERNELS[kernel], path=1, half_tiles=0).items():
        tcec.set_option(name, value)
    for m in (1, 15, 17, 33, 70, 128, 131, 300):
        for n in (1, 31, 36, 64, 67, 128, 160, 263, 288):
            a = torch.randn((m, k), generator=gen, device=DEV)
            b = torch.randn((k, n), generator=gen, device=DEV)
            p = tcec.sgemm(a, b, policy=policy)
            exact = a.double() @ b.double()
            bound = 1e-6 if policy == "fp16_ec" else 2e-3  # tf32 inputs: 2^-11 each
            assert (p.double() - exact).norm() <= bound * exact.norm(), (m, n)
            for col in (False, True):
                for pad, offset in ((0, 0), (8 - (m if col else n) % 8, 0), (3, 0), (4 - (m if col else n) % 4, 4), (1, 1)):
                    for beta in (0.0, 0.5):
                        r, c = (n, m) if col else (m, n)
                        buf = torch.full((offset + r * (c + pad),), float("nan"), device=DEV)
                        view = buf.as_strided((r, c), (c + pad, 1), offset)
                        old = torch.randn((r, c), generator=gen, device=DEV) if beta else torch.full_like(view, float("nan"))
                        view.copy_(old)
                        out = view.t() if col else view
                        tcec.sgemm(a, b, out, alpha=-2.0, beta=beta, policy=policy)
                        # powers of two: only the sum with the old value is rounded
                        want = -2.0 * p.double() + (beta * (old.t() if col else old).double() if beta else 0.0)
                        assert torch.equal(out, want.float()), (m, n, col, pad, offset, beta)
                        view.fill_(float("nan"))
                        assert torch.isnan(buf).all(), (m, n, col, pad, offset, beta)
    tcec.device_status()
