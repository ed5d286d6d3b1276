"""The split of z columns into tasks, as host code: every plane of every column
once, pieces no shorter than two planes, shares that fit the resident CTAs, and
few shares tried, since the split runs on every re-plan of a serving loop."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WENO, MUSCL, SIMPLE = 1.0, 0.65, 0.35  # plane-times of a piece's warm-up and set-up


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("split") / "split.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-shared", "-fPIC", "-o", so,
                           "-I", os.path.join(ROOT, "fvm-3d-f90_b200", "csrc"), "-I", "/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "c_driver", "fvm_split_driver.cpp")])
    return ctypes.CDLL(so)


def columns(*blocks, tx=16, ty=8):
    """The column heights of blocks (nx, ny, nz) in tiles of tx x ty."""
    return np.concatenate([np.full(-(-b[0] // tx) * -(-b[1] // ty), b[2]) for b in blocks]).astype(np.int32)


def even_split(lib, nz, slots, ovh):
    out = np.zeros((2 * len(nz) + 8 * slots, 3), np.int32)
    share, tries = ctypes.c_double(), ctypes.c_int()
    n = lib.even_split_c(len(nz), nz.ctypes.data_as(ctypes.c_void_p), slots, ctypes.c_double(ovh),
                         out.ctypes.data_as(ctypes.c_void_p), len(out), ctypes.byref(share), ctypes.byref(tries))
    assert n <= len(out)
    return out[:n], share.value, tries.value


def check_cover(tasks, nz):
    at = np.zeros(len(nz), int)
    for c, z0, z1 in tasks:
        assert z0 == at[c] and (z1 - z0 >= 2 or nz[c] < 2)
        at[c] = z1
    assert np.array_equal(at, nz)


THIN = [[(200, 200, 1)] * 300, [(33, 17, 2)] * 4000, [(1000, 1000, 2)], [(64, 64, 3)] * 500]
THICK = [[(128, 128, 128)], [(61, 83, 47)], [(20, 9, 1)], [(5, 5, 3)], [(400, 300, 24)], [(30, 30, 90), (50, 20, 7), (9, 9, 1)]]


@pytest.mark.parametrize("ovh", [WENO, MUSCL, SIMPLE])
@pytest.mark.parametrize("slots", [296, 444, 592])
@pytest.mark.parametrize("blocks", THIN + THICK, ids=lambda b: "%dx%s" % (len(b), b[0]))
def test_even_split_covers_and_fits_in_few_tries(lib, blocks, slots, ovh):
    nz = columns(*blocks)
    tasks, share, tries = even_split(lib, nz, slots, ovh)
    check_cover(tasks, nz)
    # the work with one warm-up and set-up per piece fits the CTAs' shares
    assert (tasks[:, 2] - tasks[:, 1] + ovh).sum() <= slots * share + 1e-6
    # A CTA leaves less than one least piece of its share unused (2 + ovh) and
    # cuts at most one column (another ovh): the mean and 4 plane-times more
    # always fits, 16 steps of a quarter from the first share tried.
    assert tries <= 17


def split(lib, nz, slots, prec, ovh):
    out = np.zeros((2 * len(nz) + 16 * slots, 3), np.int32)
    n = lib.split_columns_c(len(nz), nz.ctypes.data_as(ctypes.c_void_p), slots, prec, ctypes.c_double(ovh),
                            out.ctypes.data_as(ctypes.c_void_p), len(out))
    assert n <= len(out)
    return out[:n]


# The branches of the split, each with a block that takes it on 148 SMs: the
# precision form (0 exact, 1 FP64, 2 FP32), its tile, the resident CTAs of its
# kernels per SM, and what is expected. The GPU tests run the same blocks.
QUEUE, SPAN, ROUNDS, CHUNKS = "more tasks than CTAs", "shares over several columns", "two rounds", "equal chunks"
BRANCHES = [
    ((520, 300, 3), 1, (16, 8), 3, {QUEUE, SPAN}),
    ((520, 300, 3), 0, (32, 8), 2, {QUEUE, SPAN}),
    ((520, 300, 3), 2, (16, 8), 4, {QUEUE, SPAN}),
    ((520, 300, 3), 2, (32, 8), 2, {QUEUE, SPAN}),
    ((110, 110, 110), 2, (16, 8), 4, {CHUNKS}),
    ((110, 110, 110), 2, (32, 8), 2, {CHUNKS}),
    ((160, 152, 160), 1, (16, 8), 3, {QUEUE, ROUNDS}),
    ((96, 104, 128), 0, (32, 8), 2, {QUEUE, ROUNDS}),
    ((64, 48, 40), 1, (16, 8), 3, set()),
]


@pytest.mark.parametrize("ovh", [WENO, MUSCL])
@pytest.mark.parametrize("n,prec,tile,per_sm,expected", BRANCHES)
def test_every_branch_is_taken(lib, n, prec, tile, per_sm, expected, ovh):
    nz, slots = columns(n, tx=tile[0], ty=tile[1]), 148 * per_sm
    tasks = split(lib, nz, slots, prec, ovh)
    check_cover(tasks, nz)
    once, share, _ = even_split(lib, nz, slots, ovh)
    twice, _, _ = even_split(lib, nz, 2 * slots, ovh)
    got = set()
    if len(tasks) > slots:
        got.add(QUEUE)
    if share > n[2] + ovh:
        got.add(SPAN)
    if np.array_equal(tasks, twice) and not np.array_equal(once, twice):
        got.add(ROUNDS)
    if np.ptp(tasks[:, 2] - tasks[:, 1]) <= 1 and not np.array_equal(tasks, once):
        got.add(CHUNKS)
        assert len(tasks) <= slots
    if not got & {ROUNDS, CHUNKS}:
        assert np.array_equal(tasks, once)
    assert got == expected
