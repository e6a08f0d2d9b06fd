"""The complex product as one real GEMM on interleaved storage: both scalar paths, alignments, layouts and edges."""
import pytest
import torch

from wmma_extension_b200 import tcec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _view(x, layout, pad):
    """x as a row- or column-major view with `pad` complex elements between rows."""
    r, c = x.shape if layout == "r" else x.shape[::-1]
    buf = torch.full((r, c + pad), complex(float("nan"), float("nan")), dtype=torch.complex64, device=DEV)
    v = buf[:, :c]
    v.copy_(x if layout == "r" else x.t())
    return v if layout == "r" else v.t()


@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_ec"])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (3, 5, 7), (64, 64, 16), (65, 63, 17), (130, 200, 100), (300, 129, 257)])
def test_all_layouts_and_both_scalar_paths(m, n, k, policy):
    gen = torch.Generator(device=DEV).manual_seed(m * n + k)
    rnd = lambda *s: torch.complex(torch.randn(s, generator=gen, device=DEV), torch.randn(s, generator=gen, device=DEV))  # noqa: E731
    a, b, c0 = rnd(m, k), rnd(k, n), rnd(m, n)
    exact = a.to(torch.complex128) @ b.to(torch.complex128)
    for layouts in ("rrr", "rcr", "crc", "ccc"):
        A, B = _view(a, layouts[0], 1), _view(b, layouts[1], 3)
        for alpha, beta in ((1.0, 0.0), (-0.5, 0.25), (0.5 - 2j, 0.0), (1j, 0.25 + 1j)):
            C = _view(c0, layouts[2], 2)
            tcec.cgemm(A, B, C, alpha=alpha, beta=beta, policy=policy)
            tcec.device_status()
            want = alpha * exact + beta * c0.to(torch.complex128)
            # K' = 2k terms at 2^-22 relative error each way: 1e-6 of |alpha| |A| |B| is several times the worst seen
            scale = abs(alpha) * (a.abs().double() @ b.abs().double()).max() + abs(beta) * c0.abs().max()
            assert (C.to(torch.complex128) - want).abs().max() < 2e-6 * scale, (layouts, alpha, beta)


def test_operands_on_four_byte_boundaries():
    gen = torch.Generator(device=DEV).manual_seed(2)
    m, n, k = 40, 30, 50
    fa = torch.randn(2 * m * k + 1, generator=gen, device=DEV)
    fb = torch.randn(2 * k * n + 1, generator=gen, device=DEV)
    import ctypes

    one, zero = (ctypes.c_float * 2)(1, 0), (ctypes.c_float * 2)(0, 0)
    c = torch.empty((m, n), dtype=torch.complex64, device=DEV)
    st = tcec.load().tcec_cgemm(0, 0, 0, m, n, k, one, fa.data_ptr() + 4, k, fb.data_ptr() + 4, n, zero, c.data_ptr(), n, 0,
                                torch.cuda.current_stream().cuda_stream)
    assert st == tcec.OK
    tcec.device_status()
    a = torch.view_as_complex(fa[1:].clone().view(m, k, 2))
    b = torch.view_as_complex(fb[1:].clone().view(k, n, 2))
    assert torch.equal(c, tcec.cgemm(a, b))
