"""The state of blocks that take each branch of the engine's column split (which
test_split_cpu.py shows they do) against the same kernel on chunks of four
planes: bit for bit, as no cell's arithmetic depends on the tiling."""
import numpy as np
import pytest

from fvm3d import abi
from test_gpu_even_split import smooth, states
from test_split_cpu import BRANCHES

pytestmark = pytest.mark.gpu

TILES = {(32, 8): 2, (16, 8): 3}


@pytest.mark.parametrize("recon,flux", [(abi.RECON_WENO, abi.FLUX_AUSM), (abi.RECON_MUSCL, abi.FLUX_ROE)])
@pytest.mark.parametrize("n,prec,tile,per_sm,expected", BRANCHES)
def test_state_does_not_depend_on_the_branch(n, prec, tile, per_sm, expected, recon, flux):
    form = {0: abi.PREC_FP64_EXACT, 1: abi.PREC_FP64, 2: abi.PREC_FP32_FLUX}[prec]
    c = smooth([n], 3, 13, reconstruct=recon, flux_split=flux)
    ref = states(c, form, TILES[tile], 4, steps=1)[0]
    got = states(c, form, TILES[tile], 0, steps=1)[0]
    assert np.isfinite(ref).all()
    assert np.array_equal(got, ref)
