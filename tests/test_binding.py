"""The native binding of the common calls: what it does not take falls through to the Python code, with the same errors; what it
takes gives the same results."""
import importlib.util
import os
import shutil
import subprocess
import sys

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from wmma_extension_b200 import tcec

DEV = "cuda:0"


def test_it_is_built_and_leaves_other_operands_to_python():
    assert tcec._binding is not None
    x = torch.zeros(4, 4)
    assert tcec._binding.sgemm(x, x, None, 1.0, 0.0, "fp16_ec") is None  # not on a GPU
    assert tcec._binding.sgemm(x, [1], None, 1.0, 0.0, "fp16_ec") is None
    assert tcec._binding.sgemm(x) is None
    assert tcec._binding.strided(x, x, x, 1.0, 0.0, 9) is None
    assert tcec._binding.pack_a(x, "no_such_policy", None) is None
    assert tcec._binding.sgemm_packed(x, x, -1, 4, 4, None, 1.0, 0.0, 0) is None
    with pytest.raises(TypeError):
        tcec._binding.bind(1)
    tcec.load()
    for call in (lambda: tcec.sgemm(x, x), lambda: tcec.sgemm_strided_batched(x[None], x[None]), lambda: tcec.pack_a(x),
                 lambda: tcec.pack_b(x)):
        with pytest.raises(ValueError, match="float32 CUDA"):
            call()


def _another_tcec(name):
    spec = importlib.util.spec_from_file_location(f"wmma_extension_b200.{name}", tcec.__file__)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def test_a_binding_of_another_torch_is_neither_used_nor_kept(monkeypatch, tmp_path):
    import __graft_entry__ as build

    assert _another_tcec("again")._binding is tcec._binding
    tag = build._binding_tag()
    assert tcec._binding.built_for == tag
    so, source = tmp_path / "binding.so", tmp_path / "source"
    source.write_text("")
    shutil.copyfile(tcec._binding.__file__, so)
    assert build._binding_current(str(so), [str(source)], tag)
    monkeypatch.setattr(torch, "__version__", torch.__version__ + "x")
    assert not build._binding_current(str(so), [str(source)], build._binding_tag())
    assert _another_tcec("elsewhere")._binding is None


def test_the_library_is_published_after_the_binding_has_it(monkeypatch):
    """Another thread that sees the library goes straight into the binding, which then has to know the library's addresses."""
    seen = []

    class Binding:
        @staticmethod
        def bind(*addresses):
            seen.append((tcec._lib, all(addresses)))

    monkeypatch.setattr(tcec, "_lib", None)
    monkeypatch.setattr(tcec, "_binding", Binding)
    lib = tcec.load()
    assert seen == [(None, True)] and tcec._lib is lib


@pytest.mark.gpu
def test_nothing_is_called_before_bind(tmp_path):
    """A copy of the extension that nobody has bound, in a process of its own: every call is left to the Python code."""
    copy = shutil.copy(tcec._binding.__file__, tmp_path / "_binding.so")
    code = f"""
import importlib.util, torch
spec = importlib.util.spec_from_file_location("_binding", {str(copy)!r})
binding = importlib.util.module_from_spec(spec)
spec.loader.exec_module(binding)
x = torch.zeros(4, 4, device="cuda:0")
p = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda:0")
got = [binding.sgemm(x, x, None, 1.0, 0.0, 0), binding.strided(x[None], x[None], None, 1.0, 0.0, 0), binding.pack_a(x, 0, None),
       binding.pack_b(x, 0, p), binding.sgemm_packed(p, p, 4, 4, 4, None, 1.0, 0.0, 0)]
assert got == [None] * 5, got
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=120, cwd=os.path.dirname(os.path.dirname(tcec.__file__)))


@pytest.mark.gpu
def test_an_exception_out_of_the_library_leaves_the_call_to_python(tmp_path):
    """A library whose calls throw (as on a host that is out of memory), in a process of its own: the interpreter goes on, and every call
    is left to the Python code."""
    source, library = tmp_path / "throws.cpp", tmp_path / "throws.so"
    source.write_text('#include <new>\n#include <cstddef>\nextern "C" { int call(...) { throw std::bad_alloc(); } size_t bytes(int, int, int) { return 16; } }\n')
    subprocess.run(["g++", "-shared", "-fPIC", "-o", str(library), str(source)], check=True)
    copy = shutil.copy(tcec._binding.__file__, tmp_path / "_binding.so")
    code = f"""
import ctypes, importlib.util, threading, torch
lib = ctypes.CDLL({str(library)!r})
spec = importlib.util.spec_from_file_location("_binding", {str(copy)!r})
binding = importlib.util.module_from_spec(spec)
spec.loader.exec_module(binding)
call, bytes_ = (ctypes.cast(f, ctypes.c_void_p).value for f in (lib.call, lib.bytes))
binding.bind(call, call, call, call, call, bytes_)
x = torch.zeros(4, 4, device="cuda:0")
p = torch.zeros(16, dtype=torch.uint8, device="cuda:0")
def run():
    for _ in range(200):
        got = [binding.sgemm(x, x, None, 1.0, 0.0, 0), binding.strided(x[None], x[None], None, 1.0, 0.0, 0), binding.pack_a(x, 0, None),
               binding.pack_b(x, 0, p), binding.sgemm_packed(p, p, 4, 4, 4, None, 1.0, 0.0, 0)]
        assert got == [None] * 5, got
threads = [threading.Thread(target=run) for _ in range(4)]
[t.start() for t in threads]
[t.join() for t in threads]
run()
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=120, cwd=os.path.dirname(os.path.dirname(tcec.__file__)))


def _calls_without_room(dev):
    """Calls whose result, packed operands or second operand are not where or as large as the kernels would take them to be."""
    def f(*shape, device=dev):
        return torch.empty(shape, device=device)

    def u8(n, device=dev):
        return torch.empty(n, dtype=torch.uint8, device=device)

    need = 256 * 64 * 4  # 100 or 60 rows are two blocks of 128, 50 of K two of 32
    a, b, a3, b3 = f(100, 50), f(50, 60), f(4, 100, 50), f(4, 50, 60)
    return {
        "too few rows": lambda m: m.sgemm(a, b, f(10, 60)),
        "too few columns": lambda m: m.sgemm(a, b, f(100, 59)),
        "too few rows, column-major": lambda m: m.sgemm(a, b, f(60, 99).t()),
        "transposed result": lambda m: m.sgemm(a, b, f(60, 100)),
        "result of no matrices": lambda m: m.sgemm(a, b, f(0, 100, 60)),
        "complex result": lambda m: m.cgemm(*(torch.empty(s, dtype=torch.complex64, device=dev) for s in ((100, 50), (50, 60), (99, 60)))),
        "too few matrices": lambda m: m.sgemm_strided_batched(a3, b3, f(3, 100, 60)),
        "too few rows in a batch": lambda m: m.sgemm_strided_batched(a3, b3, f(4, 99, 60)),
        "one matrix for a batch": lambda m: m.sgemm_strided_batched(a3, b3, f(100, 60)),
        "no room to pack A": lambda m: m.pack_a(a, "fp16_ec", u8(need - 1)),
        "no room to pack B": lambda m: m.pack_b(b, "fp16_ec", u8(need - 1)),
        "room with holes": lambda m: m.pack_a(a, "fp16_ec", u8(2 * need)[::2]),
        "packed A too short": lambda m: m.sgemm_packed(u8(need - 1), u8(need), 100, 60, 50),
        "packed B too short": lambda m: m.sgemm_packed(u8(need), u8(need - 1), 100, 60, 50),
        "packed for another policy": lambda m: m.sgemm_packed(u8(need // 2), u8(need // 2), 100, 60, 50),
        "packed result too small": lambda m: m.sgemm_packed(u8(need), u8(need), 100, 60, 50, f(99, 60)),
        "packed operand on the host": lambda m: m.sgemm_packed(u8(need, "cpu"), u8(need), 100, 60, 50, f(100, 60)),
        "room on the host": lambda m: m.pack_a(a, "fp16_ec", u8(need, "cpu")),
        "B on the host": lambda m: m.sgemm(a, f(50, 60, device="cpu")),
    }


def _refused_before_anything_is_launched(module, call):
    with pytest.raises(ValueError, match="the result needs|consecutive bytes|one device|float32 CUDA"):
        call(module)


def test_calls_without_room_are_refused_in_python(monkeypatch):
    """Without a GPU, on stand-in tensors."""
    tcec.load()
    monkeypatch.setattr(torch.cuda, "is_available", lambda: False)  # the stand-ins' devices need not exist
    with FakeTensorMode():
        for name, call in _calls_without_room(DEV).items():
            try:
                _refused_before_anything_is_launched(tcec, call)
            except BaseException as e:
                raise AssertionError(name) from e
        a, b = torch.empty(100, 50, device=DEV), torch.empty(50, 60, device=DEV)
        packed = torch.empty(1 << 16, dtype=torch.uint8, device=DEV)
        for call in (lambda: tcec.sgemm(a, torch.empty(50, 60, device="cuda:1")),
                     lambda: tcec.sgemm(a, b, torch.empty(100, 60, device="cuda:1")),
                     lambda: tcec.pack_a(a, "fp16_ec", torch.empty(1 << 16, dtype=torch.uint8, device="cuda:1")),
                     lambda: tcec.sgemm_packed(packed, packed, 100, 60, 50, torch.empty(100, 60, device="cuda:1"))):
            with pytest.raises(ValueError, match="one device"):
                call()


@pytest.mark.gpu
def test_calls_without_room_are_refused(python_only):
    tcec.load()
    for call in _calls_without_room(DEV).values():
        _refused_before_anything_is_launched(tcec, call)
        _refused_before_anything_is_launched(python_only, call)
    # a result that is larger than the product takes it in its first rows and columns
    gen = torch.Generator(device=DEV).manual_seed(2)
    a, b = torch.rand((100, 50), generator=gen, device=DEV), torch.rand((50, 60), generator=gen, device=DEV)
    want = tcec.sgemm(a, b)
    for module in (tcec, python_only):
        for c in (torch.full((103, 64), 7.0, device=DEV), torch.full((64, 103), 7.0, device=DEV).t(), torch.full((1, 100, 60), 7.0, device=DEV)):
            assert module.sgemm(a, b, c) is c
            rest = c.clone()
            rest[..., :100, :60] = 7.0
            assert torch.equal(c[..., :100, :60].reshape(100, 60), want) and bool((rest == 7.0).all())
    tcec.device_status()


@pytest.fixture
def python_only():
    """tcec.py once more, without the binding."""
    spec = importlib.util.spec_from_file_location("tcec_python_only", tcec.__file__, submodule_search_locations=None)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)  # no package: the relative import of the binding fails
    assert module._binding is None
    return module


@pytest.mark.gpu
def test_same_results_and_errors_as_the_python_code(python_only):
    gen = torch.Generator(device=DEV).manual_seed(1)
    tcec.load()

    def rand(*shape):
        return torch.rand(shape, generator=gen, device=DEV).mul_(2).sub_(1)

    forms = {
        "row": lambda r, c: rand(r, c), "col": lambda r, c: rand(c, r).t(), "padded": lambda r, c: rand(r, c + 3)[:, :c],
        "one row": lambda r, c: rand(1, c).expand(1, c), "offset": lambda r, c: rand(r + 1, c)[1:],
    }
    for fa in forms:
        for fb in forms:
            a, b = forms[fa](33, 40), forms[fb](40, 17)
            if a.shape[1] != b.shape[0]:
                with pytest.raises(ValueError, match="inner"):
                    tcec.sgemm(a, b)
                continue
            for policy in ("fp16_ec", "tf32_ec", 2):
                assert torch.equal(tcec.sgemm(a, b, policy=policy), python_only.sgemm(a, b, policy=policy))
            c0 = rand(b.shape[1], a.shape[0]).t()
            c = [c0.clone(), c0.clone()]
            got = tcec.sgemm(a, b, c[0], alpha=0.5, beta=-1.0)
            assert got is c[0] and torch.equal(got, python_only.sgemm(a, b, c[1], alpha=0.5, beta=-1.0))
            pa, pb = tcec.pack_a(a), tcec.pack_b(b)
            assert torch.equal(pa, python_only.pack_a(a)) and torch.equal(pb, python_only.pack_b(b))
            m, n, k = a.shape[0], b.shape[1], a.shape[1]
            assert torch.equal(tcec.sgemm_packed(pa, pb, m, n, k), python_only.sgemm_packed(pa, pb, m, n, k))
    x, y = rand(3, 20, 30), rand(3, 9, 30).transpose(1, 2)
    assert torch.equal(tcec.sgemm_strided_batched(x, y), python_only.sgemm_strided_batched(x, y))
    assert tcec.sgemm(rand(0, 5), rand(5, 4)).shape == (0, 4) and tcec.sgemm(rand(4, 0), rand(0, 4)).abs().max() == 0
    for bad in (lambda m: m.sgemm(x[0], x[0]), lambda m: m.sgemm(x[0].double(), y[0]), lambda m: m.sgemm(x[0][:, ::2], y[0][::2]),
                lambda m: m.sgemm(x[0], y[0], policy="fp8"), lambda m: m.sgemm(x[0], y[0], policy=9),
                lambda m: m.sgemm(x[0], y[0], torch.zeros(20, 9, dtype=torch.float64, device=DEV)),
                lambda m: m.sgemm_strided_batched(x, y[:2]), lambda m: m.pack_a(x)):
        raised = []
        for module in (tcec, python_only):
            with pytest.raises(Exception) as e:
                bad(module)
            raised.append((type(e.value).__name__, str(e.value)))
        assert raised[0] == raised[1]
    tcec.device_status()
