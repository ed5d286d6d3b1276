"""How far one NaN cell spreads in a step: as far in the non-exact FP64 form as
in the exact one, neither less (a limiter that drops it) nor further."""
import numpy as np
import pytest

from fvm3d import abi, cases
from fvm3d.solver import FvmError, Solver

pytestmark = pytest.mark.gpu

N, AT = 48, 20


def nan_cells(prec, **cfg):
    rng = np.random.default_rng(3)
    f = lambda a, b: rng.uniform(a, b, (1, 1, N))  # noqa: E731
    q = cases.prim_to_cons(f(0.8, 1.2), f(-0.3, 0.3), f(-0.3, 0.3), f(-0.3, 0.3), f(0.8, 1.2))
    q[:, 0, 0, AT] = np.nan
    s = Solver(precision=prec, idimension=3, kappa=1.0 / 3.0, entropy_fix=0.1, rk_stages=3, timestep_set=abi.DT_FIXED,
               dt=1e-3, **cfg)
    s.add_block((N, 1, 1), (0.1, 0.1, 0.1))
    s.set_state(0, q)
    with pytest.raises(FvmError, match="NaN"):  # the residual's non-finite status
        s.step(1)
    out = np.isnan(s.get_state(0)).any(axis=0).ravel()
    s.close()
    return np.flatnonzero(out)


# three stages, each as far as the stencil of a cell's faces reaches: two cells
# of MUSCL and three of WENO5 on either side, one of the first-order form
@pytest.mark.parametrize("flux", [abi.FLUX_ROE, abi.FLUX_AUSM, abi.FLUX_VANLEER])
@pytest.mark.parametrize("recon,limiter,reach", [
    (abi.RECON_SIMPLE, abi.LIMITER_NONE, 1), (abi.RECON_MUSCL, abi.LIMITER_NONE, 2),
    (abi.RECON_MUSCL, abi.LIMITER_MINMOD, 2), (abi.RECON_MUSCL, abi.LIMITER_VANLEER, 2),
    (abi.RECON_MUSCL, abi.LIMITER_VANALBADA, 2), (abi.RECON_WENO, abi.LIMITER_NONE, 3)])
def test_one_cell_spreads_as_in_the_exact_form(recon, limiter, reach, flux):
    cfg = dict(reconstruct=recon, limiter=limiter, flux_split=flux)
    exact = nan_cells(abi.PREC_FP64_EXACT, **cfg)
    assert exact[0] >= AT - 3 * reach and exact[-1] <= AT + 3 * reach and len(exact) >= 3 * reach
    assert np.array_equal(nan_cells(abi.PREC_FP64, **cfg), exact)
