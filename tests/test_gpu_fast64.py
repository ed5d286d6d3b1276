"""The non-exact FP64 form's own arithmetic (limited slopes, Roe and AUSM
fluxes, WENO5 weights) against the oracle, for every limiter and kappa and for
supersonic and subsonic states of both signs along every axis."""
import numpy as np
import pytest

import oracle as orc
from fvm3d import abi, cases
from fvm3d.solver import Solver

pytestmark = pytest.mark.gpu

# Every flux is a few hundred operations of half an ulp on terms of the state's
# size; a step adds at most CFL times that to a cell (6 faces), three RK stages
# and three steps: below 5000 half ulps, 6e-13, of the largest component.
TOL = 1e-12


def field(n, seed, mach):
    rng = np.random.default_rng(seed)
    sh = (n[2], n[1], n[0])
    ax = [np.linspace(0, 2 * np.pi, m, endpoint=False) for m in n]
    Z, Y, X = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    w = lambda a: 1.0 + a * np.sin(X + rng.uniform(0, 6)) * np.cos(Y + rng.uniform(0, 6)) * np.cos(Z)  # noqa: E731
    vel = [mach * rng.choice([-1.0, 1.0]) * w(0.3) + 0.01 * rng.uniform(-1, 1, sh) for _ in range(3)]
    return cases.prim_to_cons(w(0.2), *vel, w(0.25) / cases.GAMMA)


@pytest.mark.parametrize("mach", [0.05, 0.9, 2.5])
@pytest.mark.parametrize("flux", [abi.FLUX_ROE, abi.FLUX_AUSM, abi.FLUX_VANLEER])
@pytest.mark.parametrize("recon,limiter,kappa,compat", [
    (abi.RECON_MUSCL, abi.SCHEME_NULL, -1.0, abi.COMPAT_REFERENCE),
    (abi.RECON_MUSCL, abi.LIMITER_NONE, 1.0 / 3.0, abi.COMPAT_REFERENCE),
    (abi.RECON_MUSCL, abi.LIMITER_MINMOD, -1.0, abi.COMPAT_REFERENCE),
    (abi.RECON_MUSCL, abi.LIMITER_VANLEER, 1.0 / 3.0, abi.COMPAT_TEXTBOOK),
    (abi.RECON_MUSCL, abi.LIMITER_VANALBADA, 0.7, abi.COMPAT_REFERENCE),
    (abi.RECON_WENO, abi.SCHEME_NULL, -1.0, abi.COMPAT_REFERENCE),
    (abi.RECON_WENO, abi.SCHEME_NULL, -1.0, abi.COMPAT_TEXTBOOK),
])
def test_fp64_form_against_oracle(recon, limiter, kappa, compat, flux, mach):
    n = (19, 10, 6)
    c = cases.Case(name="fast64", cfg=dict(idimension=3, reconstruct=recon, limiter=limiter, kappa=kappa,
                                           flux_split=flux, entropy_fix=0.1, compat=compat, rk_stages=3,
                                           timestep_set=abi.DT_CFL, cfl=0.3))
    c.blocks.append((n, (0.1, 0.12, 0.15)))
    c.origins.append((0, 0, 0))
    c.bcs = [(0, r, abi.BC_PERIODIC) for r in range(1, 7)]
    c.states.append(field(n, 7, mach))
    g = c.apply(Solver(c.config(precision=abi.PREC_FP64)))
    o = c.apply(orc.Oracle(c.config()))
    g.step(3)
    o.step(3)
    a, b = g.get_state(0), o.get_state(0)
    assert np.isfinite(b).all()
    assert np.abs(a - b).max() <= TOL * np.abs(b).max()


@pytest.mark.parametrize("limiter", [abi.LIMITER_MINMOD, abi.LIMITER_VANLEER, abi.LIMITER_VANALBADA])
@pytest.mark.parametrize("side", [-1, 1])
def test_nan_reaches_both_faces_of_a_limited_cell(limiter, side):
    # a NaN cell pollutes the same cells in one first-order-in-time stage
    # sweep as in the exact form, whichever side of a cell it is on
    n = (12, 1, 1)
    base = dict(idimension=3, reconstruct=abi.RECON_MUSCL, limiter=limiter, kappa=1.0 / 3.0,
                flux_split=abi.FLUX_ROE, entropy_fix=0.1, rk_stages=3, timestep_set=abi.DT_FIXED, dt=1e-3)
    q = field(n, 3, 0.4)
    q[:, 0, 0, 5 if side < 0 else 6] = np.nan
    got = []
    for prec in (abi.PREC_FP64_EXACT, abi.PREC_FP64):
        s = Solver(precision=prec, **base)
        s.add_block(n, (0.1, 0.1, 0.1))
        s.set_state(0, q)
        with pytest.raises(Exception):
            s.step(1)
        got.append(np.isnan(s.get_state(0)))
    assert np.array_equal(got[0], got[1])
