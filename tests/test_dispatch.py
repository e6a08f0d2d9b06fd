"""The rules that choose a kernel from sizes (csrc/tcec_dispatch.h), compiled for the host: each against what both sides were
measured to take on a B200."""
import ctypes
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("dispatch") / "dispatch.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-o", so,
                    os.path.join(ROOT, "tests", "dispatch_harness.cpp")], check=True)
    return ctypes.CDLL(so)


def _promo(k, ec):
    return 0 if not ec else 2 if k <= 2048 else 4 if k <= 4096 else 8  # K blocks of 32 per promotion


# batch, m, n, k, with error correction, us on the FP32-tile kernel, us split and from panels (strided batches)
FUSED_OR_PANELS = [
    # large matrices: conversion in every tile costs more than one split
    (2, 8192, 8192, 2048, 1, 1808, 1500), (2, 4096, 4096, 2048, 1, 437, 377), (4, 4096, 4096, 2048, 1, 886, 778),
    (4, 4096, 4096, 1024, 1, 446, 411), (8, 2048, 2048, 512, 0, 91.5, 69.0),
    # few tiles, where K runs serially in them, and three whose panels are slow all the same
    (2, 1024, 1024, 512, 1, 22.3, 15.3), (2, 1024, 1024, 1024, 1, 37.2, 21.8), (2, 1024, 1024, 2048, 1, 69.4, 37.2),
    (2, 256, 256, 256, 1, 14.6, 8.5), (2, 256, 256, 2048, 1, 73.8, 24.7), (16, 256, 256, 512, 1, 22.3, 14.4),
    (16, 256, 256, 2048, 1, 72.8, 40.2), (8, 512, 512, 2048, 1, 66.6, 47.4), (2, 64, 4096, 1024, 1, 39.7, 25.5),
    (2, 4096, 160, 2048, 1, 63.8, 47.6), (74, 36, 136, 1412, 0, 34.8, 48.3), (131, 16, 432, 356, 1, 51.2, 59.7),
    (2, 2048, 2048, 256, 1, 24.8, 28.4),
    # many matrices of a few tiles: the split is what costs
    (8192, 256, 256, 256, 1, 1290, 2400), (128, 256, 256, 256, 1, 24.8, 46.2), (128, 256, 256, 2048, 1, 128, 270),
    (1024, 160, 160, 160, 1, 75, 183), (1024, 160, 160, 1024, 1, 397, 853), (64, 400, 400, 1024, 1, 128, 174),
    (64, 512, 512, 512, 1, 67.4, 101.5), (32, 1024, 1024, 512, 1, 117, 145), (32, 1024, 1024, 1024, 1, 220, 281),
    (32, 1024, 1024, 2048, 1, 425, 488), (8, 1024, 1024, 1024, 1, 65.0, 73.9), (8, 1024, 1024, 256, 1, 23.5, 27.7),
    (8, 2048, 2048, 256, 1, 64.9, 81.0), (4, 4096, 4096, 256, 1, 126, 157), (64, 512, 136, 2048, 1, 129, 210),
    (16, 4096, 256, 1024, 1, 124, 191), (512, 64, 200, 300, 1, 75.5, 166), (64, 256, 256, 256, 0, 13.0, 19.1),
]


@pytest.mark.parametrize("case", FUSED_OR_PANELS, ids=lambda c: "x".join(map(str, c[:4])) + ("" if c[4] else "_no_ec"))
def test_batches_take_the_side_that_was_measured_faster(rules, case):
    batch, m, n, k, ec, fused_us, panels_us = case
    got = rules.fused_pays_c(m, n, k, batch, _promo(k, ec), ec, SMS, 0)
    assert bool(got) == (fused_us < panels_us)


# the same by pointer tables: us with the maps written and the panels' launches idle, us split and from panels
TABLES = [
    (2, 256, 256, 256, 23.3, 8.1), (2, 512, 512, 512, 29.3, 10.1), (2, 1024, 1024, 1024, 41.2, 20.4),
    (16, 256, 256, 128, 22.3, 8.8), (2, 4096, 4096, 512, 138.8, 126.5),
    (256, 512, 512, 512, 245, 348), (256, 512, 512, 2048, 828, 1349), (1024, 160, 160, 160, 155, 183),
    (4096, 132, 132, 132, 503, 638), (32, 1024, 1024, 2048, 406, 510),
]


@pytest.mark.parametrize("case", TABLES, ids=lambda c: "x".join(map(str, c[:4])))
def test_pointer_tables_take_the_side_that_was_measured_faster(rules, case):
    batch, m, n, k, fused_us, panels_us = case
    assert bool(rules.fused_pays_c(m, n, k, batch, _promo(k, 1), 1, SMS, 2)) == (fused_us < panels_us)


def test_the_choice_does_not_flip_back_with_more_matrices(rules):
    """One and the same matrix size: once a batch is large enough for the FP32-tile kernel, larger ones stay there, apart from
    the rounds in which a few more tiles start a new round."""
    for m, n, k in ((256, 256, 256), (512, 300, 1000), (160, 160, 2048), (1024, 1024, 512)):
        picks = [rules.fused_pays_c(m, n, k, 2 ** e, _promo(k, 1), 1, SMS, 0) for e in range(1, 16)]
        first = picks.index(1)
        assert all(picks[max(first, 8):]), (m, n, k, picks)


# batch, m, n, k, K per block, us on the direct kernel, us from panels, each one call after another (a launch more costs the
# panels up to 3 us there, which the times of longer calls, taken from graphs, have been given)
DIRECT_OR_PANELS = [
    (1, 32, 32, 32, 32, 10.2, 15.4), (1, 128, 128, 96, 32, 11.1, 15.4), (1, 128, 128, 192, 32, 13.4, 15.3),
    (1, 128, 128, 384, 32, 18.5, 14.9), (1, 128, 128, 512, 32, 21.5, 13.3), (1, 128, 128, 1024, 32, 34.8, 16.4),
    (1, 128, 128, 4096, 32, 110, 29.6), (1, 1, 128, 512, 32, 18.7, 12.3), (1, 16, 16, 1024, 32, 32.2, 16.3),
    (8, 128, 128, 128, 32, 12.1, 14.2), (8, 128, 128, 512, 32, 21.4, 13.9), (32, 128, 128, 192, 32, 13.3, 13.8),
    (32, 128, 128, 512, 32, 21.6, 17.4), (32, 128, 128, 1024, 32, 34.9, 24.6), (64, 128, 128, 512, 32, 22.3, 22.5),
    (64, 128, 128, 1024, 32, 34.9, 38.8), (64, 128, 128, 2048, 32, 71.4, 65.2), (74, 128, 128, 4096, 32, 133, 146),
    (100, 128, 128, 4096, 32, 136, 197), (100, 32, 32, 128, 32, 8.3, 11.3), (100, 32, 32, 1024, 32, 31.0, 26.0),
    (100, 32, 32, 4096, 32, 126, 78), (200, 32, 32, 1024, 32, 31.1, 41.5), (200, 32, 32, 4096, 32, 128, 147),
    (48, 64, 64, 1024, 32, 31.2, 22.3), (200, 64, 64, 4096, 32, 132, 213), (16384, 64, 64, 64, 32, 195, 1200),
    (1, 128, 128, 64, 16, 11.3, 13.2), (1, 128, 128, 192, 16, 16.4, 13.6), (1, 128, 128, 1024, 16, 53.2, 19.5),
    (32, 128, 128, 96, 16, 12.3, 13.7), (32, 128, 128, 512, 16, 30.7, 21.6), (64, 128, 128, 512, 16, 30.7, 31.7),
    (64, 128, 128, 1024, 16, 53.5, 61.4), (64, 128, 128, 4096, 16, 207, 216), (48, 128, 128, 1024, 16, 52.2, 46.3),
    (100, 32, 32, 1024, 16, 51.0, 40.8), (100, 64, 64, 1024, 16, 49.8, 51.5),
]


@pytest.mark.parametrize("case", DIRECT_OR_PANELS, ids=lambda c: "x".join(map(str, c[:4])) + ("_tf32" if c[4] == 16 else ""))
def test_small_matrices_take_the_side_that_was_measured_faster(rules, case):
    batch, m, n, k, kop, direct_us, panels_us = case
    assert bool(rules.direct_pays_c(m, n, -(-k // kop), batch, kop == 16, SMS)) == (direct_us < panels_us)


# ---------------------------------------------------------------- results that lie over operands
class Extent(ctypes.Structure):
    _fields_ = [("base", ctypes.c_void_p), ("ld", ctypes.c_longlong), ("stride", ctypes.c_longlong), ("inner", ctypes.c_int),
                ("outer", ctypes.c_int)]


def _elements(e, i):
    at = e.base // 4 + i * e.stride
    return {at + r * e.ld + j for r in range(e.outer) for j in range(e.inner)}


def _meet(c, x, batch):
    cs, xs = [_elements(c, i) for i in range(batch)], [_elements(x, i) for i in range(batch)]
    own = any(cs[i] & xs[i] for i in range(batch))
    across = any(cs[i] & xs[j] for i in range(batch) for j in range(batch) if i != j)
    return own, across


def test_no_overlap_goes_unseen(rules):
    """Every call whose result shares an element with an operand is seen, over random positions, leading dimensions and strides
    (negative and zero ones too); calls that are told apart are apart."""
    rng = random.Random(7)
    told_apart = 0
    for _ in range(20000):
        batch = rng.choice([1, 1, 2, 3, 5])
        inner, outer = rng.randrange(1, 5), rng.randrange(1, 4)
        ld = inner + rng.choice([0, 0, 1, 3, 6])
        span = (outer - 1) * ld + inner
        x = Extent(4 * rng.randrange(400, 500), ld, rng.choice([0, span, span + 2, outer * ld, 2 * outer * ld, inner, -span, 7]),
                   inner, outer)
        if rng.random() < 0.6:
            c = Extent(x.base + 4 * rng.randrange(-40, 40), ld, x.stride, rng.randrange(1, ld + 1), rng.randrange(1, 4))
        else:
            i2 = rng.randrange(1, 5)
            c = Extent(x.base + 4 * rng.randrange(-40, 40), i2 + rng.randrange(0, 4), rng.choice([0, 3, 9, 20, -12]), i2,
                       rng.randrange(1, 4))
        own, across = _meet(c, x, batch)
        got = rules.batch_overlap_c(ctypes.byref(c), ctypes.byref(x), batch)
        assert (not own or got & 1) and (not across or got & 2), [(e.base, e.ld, e.stride, e.inner, e.outer) for e in (c, x)]
        told_apart += got == 0
        if batch == 1:
            one = rules.matrices_may_overlap_c(ctypes.byref(c), ctypes.byref(x))
            assert one or not own
    assert told_apart > 4000


@pytest.mark.parametrize("what,c,x,batch,want", [
    ("apart", Extent(8192, 8, 64, 8, 8), Extent(4096, 8, 64, 8, 8), 16, 0),
    ("in place", Extent(4096, 8, 64, 8, 8), Extent(4096, 8, 64, 8, 8), 16, 1),
    ("in place, padded", Extent(4096, 10, 100, 8, 8), Extent(4096, 10, 100, 8, 8), 16, 1),
    ("one matrix on", Extent(4096 + 256, 8, 64, 8, 8), Extent(4096, 8, 64, 8, 8), 16, 2),
    ("alternating matrices", Extent(4096 + 256, 8, 128, 8, 8), Extent(4096, 8, 128, 8, 8), 16, 0),
    ("column blocks of one matrix", Extent(4096 + 32, 24, 24 * 8, 8, 8), Extent(4096, 24, 24 * 8, 8, 8), 16, 0),
    ("one operand for all, result over it", Extent(4096, 8, 64, 8, 8), Extent(4096, 8, 0, 8, 8), 16, 3),
    ("single product in place", Extent(4096, 8, 0, 8, 8), Extent(4096, 8, 0, 8, 8), 1, 1),
    ("strides near the end of 64 bits", Extent(4096, 8, 2 ** 61, 8, 8), Extent(2 ** 40, 8, -2 ** 61, 8, 8), 2 ** 30, 3),
], ids=lambda v: v if isinstance(v, str) else "")
def test_usual_forms_are_told_apart(rules, what, c, x, batch, want):
    assert rules.batch_overlap_c(ctypes.byref(c), ctypes.byref(x), batch) == want


SLOTS = (ctypes.c_int * 3)(74, 33, 15)  # clusters of 2, 4, 8 CTAs that run at a time

# m, n, k, K per block, with error correction, the number of parts that was measured fastest
PARTS = [
    (64, 4096, 4096, 32, 1, 4), (33, 206, 11446, 32, 1, 8), (110, 1161, 3881, 32, 1, 8), (813, 1122, 3183, 32, 1, 2),
    (16, 8182, 3244, 32, 1, 2), (344, 402, 2524, 32, 0, 8), (632, 538, 5451, 16, 1, 4), (187, 1155, 9382, 32, 0, 4),
    (77, 6331, 1115, 32, 1, 1), (1747, 274, 1502, 32, 0, 1), (35, 3250, 795, 32, 1, 1), (4096, 4096, 4096, 32, 1, 1),
]


@pytest.mark.parametrize("case", PARTS, ids=lambda c: "x".join(map(str, c[:3])))
def test_k_is_divided_as_was_measured_fastest(rules, case):
    m, n, k, kop, ec, parts = case
    nkb = -(-k // kop)
    assert rules.divide_k_c(m, n, k, 1, nkb, ec, SLOTS, -1) == parts
    assert rules.divide_k_c(m, n, k, 1, nkb, ec, SLOTS, 1) == 1
    assert rules.divide_k_c(m, n, k, 2, nkb, ec, SLOTS, -1) == 1  # batches stay whole
    assert rules.divide_k_c(m, n, k, 1, nkb, ec, (ctypes.c_int * 3)(), -1) == 1  # nowhere to divide


def test_parts_follow_from_sizes_alone(rules):
    """GPUs differ in how many clusters they run at a time (a GPC may lack SMs); results do not."""
    rng = random.Random(11)
    gpus = [(ctypes.c_int * 3)(*s) for s in ((74, 37, 18), (74, 35, 16), (74, 33, 15), (70, 30, 12), (1, 1, 1))]
    seen = set()
    for _ in range(3000):
        m, n, k, ec = rng.randrange(1, 3000), rng.randrange(1, 3000), rng.randrange(1000, 9000), rng.randrange(2)
        for forced in (-1, 2, 4, 8):
            parts = {rules.divide_k_c(m, n, k, 1, -(-k // 32), ec, s, forced) for s in gpus}
            assert len(parts) == 1, (m, n, k, forced)
            seen |= parts
    assert seen == {1, 2, 4, 8}


def test_a_part_has_a_k_block_and_a_cluster_has_room(rules):
    for forced in (2, 4, 8):
        assert rules.divide_k_c(200, 200, 96, 1, forced - 1, 1, SLOTS, forced) == 1
        assert rules.divide_k_c(200, 200, 96, 1, forced, 1, SLOTS, forced) == forced
    assert rules.divide_k_c(128, 128 * 16, 4000, 1, 125, 1, SLOTS, 8) == 1  # 16 tiles, 15 clusters of 8
    assert rules.divide_k_c(100, 128, 4000, 1, 125, 1, SLOTS, 8) == 1  # one tile


def test_pairs_and_pacing(rules):
    for m, n, k, ec, pays in ((16384, 16384, 16384, 1, 1), (8192, 8192, 8192, 1, 1), (1000, 1000, 1000, 1, 1), (300, 16384, 65536, 0, 1),
                              (300, 16384, 65536, 1, 0), (128 * 19, 16384, 16384, 1, 1)):
        assert rules.pairs_pay_c(m, n, k, 1, ec) == pays, (m, n, k, ec)
    for m, n, k, images, paced in ((16384, 16384, 16384, 2, 1), (8192, 8192, 8192, 2, 1), (12000, 4000, 12000, 2, 1), (4096, 4096, 4096, 2, 0),
                                   (16384, 16384, 16384, 1, 1), (8192, 8192, 8192, 1, 0), (534, 8189, 3656, 2, 0)):
        assert rules.pace_pays_c(m, n, 1, -(-k // 32), images, 74) == paced, (m, n, k, images)


def test_long_calls_with_correction_draw_their_tiles(rules):
    for m, n, k, ec, draws in ((16384, 16384, 16384, 1, 1), (8192, 8192, 4096, 1, 1), (40000, 50000, 64, 1, 1), (4096, 4096, 4096, 1, 0),
                               (2048, 2048, 60000, 1, 0), (8192, 8192, 8192, 0, 0)):
        assert rules.draws_pay_c(m, n, k, ec, 74) == draws, (m, n, k, ec)
