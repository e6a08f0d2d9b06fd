"""The direct kernel (FP32 operands split on the way into shared memory, one launch) against the operand-panel path:
the same bits over every form of operand that it accepts."""
import pytest
import torch

from wmma_extension_b200 import tcec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _default_options():
    yield
    for name, value in (("direct_kernel", -1), ("path", 0), ("cta_pair", -1)):
        tcec.set_option(name, value)


def _operand(gen, batch, rows, cols, layout, pad, offset):
    """batch x rows x cols view: row- or column-major, `pad` elements between rows, base `offset` elements off 16 bytes."""
    r, c = (rows, cols) if layout == "r" else (cols, rows)
    ld = c + pad
    stride = r * ld + pad
    buf = torch.full((offset + batch * stride,), float("nan"), device=DEV)
    v = buf.as_strided((batch, r, c), (stride, ld, 1), offset)
    v.copy_(torch.rand((batch, r, c), generator=gen, device=DEV).mul_(2).sub_(1))
    return buf, (v if layout == "r" else v.transpose(1, 2))


def _run(direct, a, b, c, alpha, beta, policy, lists):
    tcec.set_option("direct_kernel", 1 if direct else 0)
    tcec.set_option("path", 0 if direct else 1)
    if lists:
        tcec.sgemm_batched(list(a), list(b), list(c), alpha=alpha, beta=beta, policy=policy)
    elif a.shape[0] == 1:
        tcec.sgemm(a[0], b[0], c[0], alpha=alpha, beta=beta, policy=policy)
    else:
        tcec.sgemm_strided_batched(a, b, c, alpha=alpha, beta=beta, policy=policy)
    tcec.device_status()


@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_ec", "fp16_no_ec", "tf32_no_ec"])
@pytest.mark.parametrize("m,n,k,batch", [
    (1, 1, 1, 1), (32, 32, 32, 1), (33, 17, 15, 7), (32, 32, 16, 9), (31, 5, 97, 5), (64, 64, 64, 5), (64, 33, 65, 2),
    (63, 64, 31, 300), (65, 1, 33, 3), (128, 128, 128, 2), (128, 120, 17, 1), (129, 128, 64, 3), (127, 257, 200, 2),
    (300, 140, 130, 160), (16, 300, 129, 4),
])
def test_same_bits_as_the_panel_path(m, n, k, batch, policy):
    gen = torch.Generator(device=DEV).manual_seed(m * 7919 + n * 31 + k)
    forms = [("r", "r", "r", 0, 0), ("r", "c", "c", 4, 0), ("c", "r", "r", 3, 1), ("c", "c", "c", 0, 2), ("r", "c", "r", 1, 3)]
    for la, lb, lc, pad, offset in forms:
        _, a = _operand(gen, batch, m, k, la, pad, offset)
        _, b = _operand(gen, batch, k, n, lb, pad, offset)
        cbuf, c = _operand(gen, batch, m, n, lc, pad, offset)
        for alpha, beta, lists in ((1.0, 0.0, False), (-0.5, 0.75, batch > 1)):
            before = cbuf.clone()
            _run(False, a, b, c, alpha, beta, policy, lists)
            want = cbuf.clone()
            cbuf.copy_(before)
            _run(True, a, b, c, alpha, beta, policy, lists)
            what = (la, lb, lc, pad, offset, alpha, beta)
            assert torch.equal(cbuf.nan_to_num(7e30), want.nan_to_num(7e30)), what  # the padding is NaN before and after
            cbuf.copy_(before)


def _strided(gen, batch, rows, cols, k_contiguous, pad, stride_pad, is_b):
    """Operand of which K is contiguous or not, `pad` elements after each row of memory, `stride_pad` after each matrix; stride_pad None: one
    matrix for all."""
    r, c = (rows, cols) if k_contiguous != is_b else (cols, rows)
    ld = c + pad
    stride = 0 if stride_pad is None else r * ld + stride_pad
    buf = torch.rand(((batch - 1) * stride + r * ld,), generator=gen, device=DEV).mul_(2).sub_(1)
    v = buf.as_strided((batch, r, c), (stride, ld, 1))
    return v if k_contiguous != is_b else v.transpose(1, 2)


# Three or more tiles a CTA, so that a lane's pointers are carried from tile to tile, and a last tile that is not full.
@pytest.mark.parametrize("m,n,k,per_tile", [
    (32, 32, 32, 4), (20, 31, 40, 4), (31, 32, 33, 4), (64, 64, 64, 2), (50, 40, 100, 2), (33, 64, 31, 2), (128, 128, 64, 1), (100, 127, 36, 1),
    (65, 128, 97, 1),
])
@pytest.mark.parametrize("policy", ["fp16_ec", "tf32_ec"])
def test_pointers_carried_over_many_tiles(m, n, k, per_tile, policy):
    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    batch = per_tile * 148 * 3 + (per_tile + 1) // 2  # the last tile holds half of what it could
    # pad to a leading dimension that is a multiple of 4 or not, and to a stride that is or not; for A and B alike and crossed
    def pads(ka, kb):
        ca, cb = (k if ka else m), (k if kb else n)
        for ld4_a, s4_a, ld4_b, s4_b in ((1, 1, 1, 1), (1, 0, 1, 1), (1, 1, 1, 0), (0, 0, 1, 1), (1, 1, 0, 0), (0, 1, 0, 1), (1, None, 1, 1),
                                         (1, 1, 1, None), (0, None, 0, None)):
            def pad(cols, ld4):
                return -cols % 4 if ld4 else (1 if (cols + 1) % 4 else 2)
            def extra(s4):
                return None if s4 is None else 4 if s4 else 1
            yield pad(ca, ld4_a), extra(s4_a), pad(cb, ld4_b), extra(s4_b)

    for ka in (True, False):
        for kb in (True, False):
            for pa, sa, pb, sb in pads(ka, kb):
                a = _strided(gen, batch, m, k, ka, pa, sa, False)
                b = _strided(gen, batch, k, n, kb, pb, sb, True)
                c = torch.full((batch, m, n), float("nan"), device=DEV)
                _run(False, a, b, c, 1.0, 0.0, policy, False)
                want = c.clone()
                c.fill_(float("nan"))
                _run(True, a, b, c, 1.0, 0.0, policy, False)
                assert torch.equal(c, want), (ka, kb, pa, sa, pb, sb)


def test_non_finite_operands_stay_in_their_rows_and_columns():
    gen = torch.Generator(device=DEV).manual_seed(3)
    for m, n, batch in ((40, 40, 6), (20, 30, 9), (100, 90, 2)):
        a = torch.randn((batch, m, 50), generator=gen, device=DEV)
        b = torch.randn((batch, 50, n), generator=gen, device=DEV)
        a[1, 3, 5] = float("nan")
        b[0, 7, 2] = float("inf")
        c = torch.empty((batch, m, n), device=DEV)
        _run(True, a, b, c, 1.0, 0.0, "tf32_ec", False)
        bad = ~torch.isfinite(c)
        want = torch.zeros_like(bad)
        want[1, 3, :] = True
        want[0, :, 2] = True
        assert torch.equal(bad, want)


def test_pointer_tables_that_mix_alignments():
    """Whether 16-byte loads may be used is decided per matrix."""
    gen = torch.Generator(device=DEV).manual_seed(4)
    m, n, k, batch = 60, 50, 70, 6
    pool = torch.rand((3, batch * 8000), generator=gen, device=DEV)
    off = [0, 1, 2, 3, 4, 5]
    lda, ldb = 72, 72  # K contiguous on both sides
    a = [pool[0].as_strided((m, k), (lda, 1), 8000 * i + off[i]) for i in range(batch)]
    b = [pool[1].as_strided((k, n), (1, ldb), 8000 * i + off[i]) for i in range(batch)]
    out = []
    for direct in (False, True):
        c = [torch.empty((m, n), device=DEV) for _ in range(batch)]
        tcec.set_option("direct_kernel", 1 if direct else 0)
        tcec.set_option("path", 0 if direct else 1)
        tcec.sgemm_batched(a, b, c)
        out.append(torch.stack(c))
    tcec.device_status()
    assert torch.equal(out[0], out[1])


def test_runs_under_graph_capture_and_on_other_streams():
    """The route allocates nothing, so a first call may be captured; streams do not share anything."""
    gen = torch.Generator(device=DEV).manual_seed(5)
    a = torch.randn((200, 48, 56), generator=gen, device=DEV)
    b = torch.randn((200, 56, 40), generator=gen, device=DEV)
    want = tcec.sgemm_strided_batched(a, b)
    c = torch.zeros_like(want)
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        tcec.sgemm_strided_batched(a, b, c)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(c, want)
    streams = [torch.cuda.Stream() for _ in range(3)]
    outs = [torch.zeros_like(want) for _ in streams]
    torch.cuda.synchronize()
    for _ in range(3):
        for st, o in zip(streams, outs):
            with torch.cuda.stream(st):
                tcec.sgemm_strided_batched(a, b, o)
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
    tcec.device_status()
