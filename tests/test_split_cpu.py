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
