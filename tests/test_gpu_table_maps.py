"""Batches by pointer tables through the FP32-tile kernel (tensor maps written on the GPU) and, where a pointer is not
16-byte aligned, through the panel kernels launched behind it: the bits of the panel path either way."""
import pytest
import torch

from wmma_extension_b200 import tcec

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _default_options():
    yield
    tcec.set_option("path", 0)


def _matrices(gen, batch, rows, cols, layout, ld, offsets):
    """`batch` rows x cols views with leading dimension `ld`, matrix i starting offsets[i % len] elements off 16 bytes."""
    r, c = (rows, cols) if layout == "r" else (cols, rows)
    pitch = r * ld + 8
    pool = torch.rand(batch * pitch + 8, generator=gen, device=DEV).mul_(2).sub_(1)
    out = []
    for i in range(batch):
        v = pool.as_strided((r, c), (ld, 1), i * pitch // 4 * 4 + offsets[i % len(offsets)])
        out.append(v if layout == "r" else v.t())
    return out


@pytest.mark.parametrize("policy", ["fp16_ec", "fp16_no_ec"])
@pytest.mark.parametrize("m,n,k,batch,offsets", [
    (130, 132, 36, 3, [0]), (256, 256, 64, 90, [0]), (512, 300, 160, 40, [0]), (37, 260, 500, 4, [0]), (300, 140, 1030, 3, [0]),
    (130, 132, 36, 5, [0, 0, 1]), (256, 256, 64, 90, [2]), (300, 140, 130, 5, [0, 3]),
    (37, 132, 20, 801, [0, 0, 0, 2]),  # an odd number of panels, more than the split's CTAs draw at first
])
def test_same_bits_as_the_panel_path(m, n, k, batch, offsets, policy):
    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    up = lambda x: (x + 3) // 4 * 4 + 4  # noqa: E731
    for la, lb, lc in (("r", "c", "c"), ("r", "r", "r"), ("c", "c", "r")):
        a = _matrices(gen, batch, m, k, la, up(k if la == "r" else m), offsets)
        b = _matrices(gen, batch, k, n, lb, up(n if lb == "r" else k), offsets)
        c0 = _matrices(gen, batch, m, n, lc, (n if lc == "r" else m) + 1, [0, 1])
        for alpha, beta in ((1.0, 0.0), (-0.5, 0.75)):
            out = []
            for path in (1, 2):  # 2: automatic takes panels for calls as short as these
                tcec.set_option("path", path)
                c = [x.clone() for x in c0]
                tcec.sgemm_batched(a, b, c, alpha=alpha, beta=beta, policy=policy)
                tcec.device_status()
                out.append(torch.stack(c))
            assert torch.equal(out[0], out[1]), (la, lb, lc, alpha, beta)


def test_tables_that_change_between_replays_of_a_graph():
    """The maps are written by the call, not kept: a captured call follows its tables, to unaligned matrices too."""
    gen = torch.Generator(device=DEV).manual_seed(6)
    m = n = k = 160
    batch = 5
    a = [_matrices(gen, batch, m, k, "r", k, [o]) for o in (0, 0, 1)]
    b = [_matrices(gen, batch, k, n, "c", k, [o]) for o in (0, 0, 1)]
    want = [torch.stack([tcec.sgemm(x, y) for x, y in zip(p, q)]) for p, q in zip(a, b)]
    tcec.set_option("path", 2)
    c = [torch.empty((m, n), device=DEV) for _ in range(batch)]
    ptrs = lambda ts: torch.tensor([t.data_ptr() for t in ts], dtype=torch.int64, device=DEV)  # noqa: E731
    pa, pb, pc = ptrs(a[0]), ptrs(b[0]), ptrs(c)

    def call():
        st = tcec.load().tcec_sgemm_batched(0, 1, 0, m, n, k, 1.0, pa.data_ptr(), k, pb.data_ptr(), k, 0.0, pc.data_ptr(), n,
                                            batch, 0, torch.cuda.current_stream().cuda_stream)
        assert st == tcec.OK

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        call()  # the workspace exists before the capture
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        call()
    for i in (0, 1, 2, 0):
        pa.copy_(ptrs(a[i]))
        pb.copy_(ptrs(b[i]))
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(torch.stack(c), want[i]), i
    tcec.device_status()
