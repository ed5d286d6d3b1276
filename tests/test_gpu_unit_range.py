"""The Euler equations keep their form when density and pressure, velocity and
length are scaled by powers of two, and so does every operation of the sweep:
a state in other units evolves into the same numbers in those units. The
powers here put density and pressure where their product leaves the range of
FP64 while each of them, and every flux, is an ordinary number."""
import numpy as np
import pytest

from fvm3d import abi, cases
from fvm3d.solver import Solver

pytestmark = pytest.mark.gpu

N = (19, 10, 6)


def evolve(mass_exp, prec, steps=3, **cfg):
    """The state after `steps` steps with mass and length scaled by 2^mass_exp (velocities and residuals are not)."""
    rng = np.random.default_rng(7)
    sh = (N[2], N[1], N[0])
    f = lambda a, b: rng.uniform(a, b, sh)  # noqa: E731
    q = cases.prim_to_cons(f(0.8, 1.2), f(-1.5, 1.5), f(-1.5, 1.5), f(-1.5, 1.5), f(0.5, 1.0))
    s = Solver(precision=prec, idimension=3, entropy_fix=0.1, rk_stages=3, timestep_set=abi.DT_CFL, cfl=0.2, **cfg)
    s.add_block(N, tuple(np.ldexp(h, mass_exp) for h in (0.1, 0.12, 0.15)))
    s.set_state(0, np.ldexp(q, mass_exp))
    s.step(steps)
    out = np.ldexp(s.get_state(0), -mass_exp)
    s.close()
    return out


# At 2^-530 the product of density and pressure is below the normal range, at
# 2^520 it overflows. Whatever formula the flux takes there, a few hundred
# operations of half an ulp per step and component, three stages and three
# steps, stay below 5000 half ulps, 6e-13, of the largest component.
@pytest.mark.parametrize("exp", [-530, 520])
@pytest.mark.parametrize("recon", [abi.RECON_SIMPLE, abi.RECON_MUSCL])
def test_ausm_where_density_times_pressure_leaves_the_range(recon, exp):
    cfg = dict(reconstruct=recon, limiter=abi.LIMITER_NONE, kappa=1.0 / 3.0, flux_split=abi.FLUX_AUSM)
    ref, got = evolve(0, abi.PREC_FP64, **cfg), evolve(exp, abi.PREC_FP64, **cfg)
    assert np.isfinite(ref).all() and np.isfinite(got).all()
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


# Differences of neighbouring cells of 1e-160 have a product that underflows;
# minmod compares magnitudes and signs and does not multiply. Every operation
# of this sweep scales exactly.
@pytest.mark.parametrize("prec", [abi.PREC_FP64_EXACT, abi.PREC_FP64])
def test_minmod_slopes_of_small_differences(prec):
    cfg = dict(reconstruct=abi.RECON_MUSCL, limiter=abi.LIMITER_MINMOD, kappa=1.0 / 3.0,
               flux_split=abi.FLUX_VANLEER)
    ref, got = evolve(0, prec, **cfg), evolve(-560, prec, **cfg)
    assert np.isfinite(ref).all()
    assert np.array_equal(got, ref)
