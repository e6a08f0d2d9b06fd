"""The bounded waits of the kernels, made to run out on purpose - by a stall made on the host side
of the launch, never by a fault: a build of the library with a short wait limit is told (through a
development switch that only that build has) to leave one ring stage unfilled, so the MMA thread's
wait gives up, every role of every CTA returns, and the host reads TCEC_ERR_TIMEOUT.  The context
stays usable: the next call gives correct results."""
import ctypes
import os

import numpy as np
import pytest
import torch

from oracle import cpu

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TEST_LIB = os.path.join(ROOT, "tests", "_build", "libtcec_b200_shortwait.so")
ERR_TIMEOUT = 4


def _library():
    if not os.path.exists(TEST_LIB):
        pytest.skip("the short-wait test build of the library is missing (run build())")
    lib = ctypes.CDLL(TEST_LIB)
    i, ll, f, p = ctypes.c_int, ctypes.c_longlong, ctypes.c_float, ctypes.c_void_p
    lib.tcec_sgemm.argtypes = [i, i, i, i, i, i, f, p, ll, p, ll, f, p, ll, i, p]
    lib.tcec_device_status.argtypes = [ctypes.POINTER(i)]
    lib.tcec_set_option.argtypes = [ctypes.c_char_p, i]
    return lib


def test_a_wait_that_runs_out_is_reported_and_leaves_the_context_usable():
    lib, i = _library(), ctypes.c_int
    rng = np.random.default_rng(3)
    m, n, k = 128, 256, 512  # one tile, 16 K blocks: more than the ring holds
    a = torch.from_numpy(rng.uniform(-1, 1, (m, k)).astype(np.float32)).cuda()
    b = torch.from_numpy(rng.uniform(-1, 1, (k, n)).astype(np.float32)).cuda()
    c = torch.zeros((m, n), device="cuda")

    def run():
        return lib.tcec_sgemm(0, 0, 0, m, n, k, 1.0, a.data_ptr(), k, b.data_ptr(), n, 0.0, c.data_ptr(), n, 0, None)

    detail = i(0)
    assert lib.tcec_set_option(b"path", 1) == 0
    assert run() == 0 and lib.tcec_device_status(ctypes.byref(detail)) == 0  # the build works
    assert lib.tcec_set_option(b"debug_flags", 32) == 0  # one stage is never filled
    try:
        assert run() == 0  # the launch itself succeeds
        st = lib.tcec_device_status(ctypes.byref(detail))
    finally:
        lib.tcec_set_option(b"debug_flags", 0)
    assert st == ERR_TIMEOUT, st
    assert detail.value in (1, 2, 3)  # which role gave up first (producer, MMA thread or epilogue)
    assert lib.tcec_device_status(ctypes.byref(detail)) == 0  # reading the status clears it
    # the context is intact: a normal call gives the right answer
    c.fill_(float("nan"))
    assert run() == 0 and lib.tcec_device_status(ctypes.byref(detail)) == 0
    exact = cpu.gemm_f64(a.cpu().numpy(), b.cpu().numpy())
    assert cpu.errors(c.cpu().numpy(), exact)["max_rel"] < 1e-6
    lib.tcec_destroy()


@pytest.mark.parametrize("policy", [0, 1, 2, 3])
@pytest.mark.parametrize("kernel", ["direct", "narrow 32", "narrow 64", "narrow 128"])
def test_waits_of_the_direct_and_narrow_kernels_run_out_the_same_way(kernel, policy):
    """Both accumulators exist twice there, and the direct kernel's stages are filled by eight warps (with tf32 two stages
    at a time), so their ways out are their own."""
    lib, i = _library(), ctypes.c_int
    rng = np.random.default_rng(4)
    m, n, k = 120, 128, 1100  # more K blocks than any ring holds, and a last one that is not whole
    a = torch.from_numpy(rng.uniform(-1, 1, (m, k)).astype(np.float32)).cuda()
    b = torch.from_numpy(rng.uniform(-1, 1, (k, n)).astype(np.float32)).cuda()
    c = torch.zeros((m, n), device="cuda")
    detail = i(0)

    def run():
        st = lib.tcec_sgemm(0, 0, 0, m, n, k, 1.0, a.data_ptr(), k, b.data_ptr(), n, 0.0, c.data_ptr(), n, policy, None)
        return st or lib.tcec_device_status(ctypes.byref(detail))

    options = {b"path": 0, b"direct_kernel": 1 if kernel == "direct" else 0,
               b"narrow_tiles": -1 if kernel == "direct" else int(kernel.split()[1])}
    for name, value in options.items():
        assert lib.tcec_set_option(name, value) == 0
    try:
        assert run() == 0
        want = c.clone()
        assert lib.tcec_set_option(b"debug_flags", 64) == 0  # one stage is never filled
        assert run() == ERR_TIMEOUT
        assert detail.value in (1, 2, 3)
        assert lib.tcec_set_option(b"debug_flags", 0) == 0
        c.fill_(float("nan"))
        assert run() == 0  # the status was cleared, TMEM and barriers are there again
        assert torch.equal(c, want)
    finally:
        for name, value in ((b"debug_flags", 0), (b"direct_kernel", -1), (b"narrow_tiles", -1)):
            lib.tcec_set_option(name, value)
        lib.tcec_destroy()


@pytest.mark.parametrize("policy", [0, 1, 2, 3])
@pytest.mark.parametrize("parts", [2, 4, 8])
def test_a_tile_of_which_one_part_is_missing_is_not_stored(parts, policy):
    """Of the CTAs that share a tile's K one gives up; the others have their parts, and still none of the tile is written."""
    lib, i = _library(), ctypes.c_int
    rng = np.random.default_rng(5)
    m, n, k = 130, 250, 8 * 32 * 11  # a part has more K blocks than the ring, whatever the policy
    a = torch.from_numpy(rng.uniform(-1, 1, (m, k)).astype(np.float32)).cuda()
    b = torch.from_numpy(rng.uniform(-1, 1, (k, n)).astype(np.float32)).cuda()
    c = torch.full((m, n), 5.0, device="cuda")
    detail = i(0)

    def run():
        st = lib.tcec_sgemm(0, 0, 0, m, n, k, 1.0, a.data_ptr(), k, b.data_ptr(), n, 0.0, c.data_ptr(), n, policy, None)
        return st or lib.tcec_device_status(ctypes.byref(detail))

    assert lib.tcec_set_option(b"k_parts", parts) == 0
    try:
        assert run() == 0
        want = c.clone()
        assert not bool((want == 5.0).any())
        assert lib.tcec_set_option(b"debug_flags", 64) == 0  # one stage of one part is never filled
        c.fill_(5.0)
        assert run() == ERR_TIMEOUT
        assert detail.value in (1, 2, 3)
        assert bool((c == 5.0).all())
        assert lib.tcec_set_option(b"debug_flags", 0) == 0
        assert run() == 0 and torch.equal(c, want)
    finally:
        for name, value in ((b"debug_flags", 0), (b"k_parts", -1)):
            lib.tcec_set_option(name, value)
        lib.tcec_destroy()


@pytest.mark.parametrize("policy", [0, 1, 2, 3])
@pytest.mark.parametrize("long", [False, True])
def test_waits_of_the_pair_kernel_run_out_the_same_way(long, policy):
    """Both CTAs of a pair leave; with correction a long call draws its tiles, and the counter is back at zero for the next one."""
    lib, i = _library(), ctypes.c_int
    m, n, k = (5000, 5000, 5200) if long else (300, 600, 1100)
    gen = torch.Generator(device="cuda").manual_seed(6)
    a, b = torch.rand((m, k), generator=gen, device="cuda"), torch.rand((k, n), generator=gen, device="cuda")
    c = torch.zeros((m, n), device="cuda")
    detail = i(0)

    def run():
        st = lib.tcec_sgemm(0, 0, 0, m, n, k, 1.0, a.data_ptr(), k, b.data_ptr(), n, 0.0, c.data_ptr(), n, policy, None)
        return st or lib.tcec_device_status(ctypes.byref(detail))

    for name, value in ((b"cta_pair", 1), (b"half_tiles", 0)):
        assert lib.tcec_set_option(name, value) == 0
    try:
        # the short limit of this build is no longer than a long call's waits, so it may run out by itself there
        healthy = run()
        assert healthy in ((0, ERR_TIMEOUT) if long else (0,))
        want = c.clone()
        assert lib.tcec_set_option(b"debug_flags", 32) == 0  # one stage of every CTA is never filled
        assert run() == ERR_TIMEOUT
        assert detail.value in (1, 2, 3)
        assert lib.tcec_set_option(b"debug_flags", 0) == 0
        again = run()
        assert again in ((0, ERR_TIMEOUT) if long else (0,))
        assert torch.equal(c, want) or healthy or again
    finally:
        for name, value in ((b"debug_flags", 0), (b"cta_pair", -1), (b"half_tiles", 1)):
            lib.tcec_set_option(name, value)
        lib.tcec_destroy()
