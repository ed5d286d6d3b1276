"""The engine's own split of z columns over the resident CTAs against fixed
z chunks: the state must not depend on it, in any form, for any block shape,
alone, over several blocks and in a batch, and one plane per task in 2D."""
import numpy as np
import pytest

from fvm3d import abi, cases, tuning
from fvm3d.solver import Solver

pytestmark = pytest.mark.gpu

FORMS = [abi.PREC_FP64_EXACT, abi.PREC_FP64, abi.PREC_FP32_FLUX]


def smooth(shapes, idim, seed, **cfg):
    rng = np.random.default_rng(seed)
    c = cases.Case(name="split", cfg=dict(idimension=idim, rk_stages=3, timestep_set=abi.DT_CFL, cfl=0.4,
                                          entropy_fix=0.1, kappa=1.0 / 3.0, limiter=abi.LIMITER_VANLEER, **cfg))
    for n in shapes:
        sh = (n[2], n[1], n[0])
        f = lambda a, b: rng.uniform(a, b, sh)  # noqa: E731
        c.blocks.append((tuple(n), (0.1, 0.1, 0.1)))
        c.states.append(cases.prim_to_cons(f(0.9, 1.1), f(-0.3, 0.3), f(-0.3, 0.3), f(-0.3, 0.3), f(0.9, 1.1)))
        c.origins.append((0, 0, 0))
    return c


def states(c, prec, tile, zchunk, steps=2):
    s = Solver(c.config(precision=prec))
    c.apply(s)
    if tile is not None:
        tuning.set_tuning(s, 0, tile, zchunk)
    s.step(steps)
    out = [s.get_state(b) for b in range(len(c.blocks))]
    s.close()
    return out


# nz of 1, 2 and 3 (shorter than a piece, one short piece), columns that are
# cut in the middle, more columns than CTAs, and blocks of different heights
SHAPES = [[(20, 9, 1)], [(17, 8, 2)], [(5, 5, 3)], [(33, 17, 29)], [(61, 40, 13)], [(150, 130, 5)],
          [(16, 8, 200)], [(48, 33, 7), (20, 20, 40), (9, 9, 1), (70, 16, 11)]]


@pytest.mark.parametrize("prec", FORMS)
@pytest.mark.parametrize("recon,flux,tile", [(abi.RECON_WENO, abi.FLUX_AUSM, 3), (abi.RECON_MUSCL, abi.FLUX_ROE, 3),
                                             (abi.RECON_SIMPLE, abi.FLUX_VANLEER, 3)])
@pytest.mark.parametrize("shapes", SHAPES)
def test_split_does_not_change_state(shapes, recon, flux, tile, prec):
    c = smooth(shapes, 3, 11, reconstruct=recon, flux_split=flux)
    if prec == abi.PREC_FP64_EXACT:
        tile = 2 if min(n[0] for n, _ in c.blocks) >= 32 else 1  # the same kernel as the engine's choice
    elif prec == abi.PREC_FP32_FLUX and recon == abi.RECON_WENO:
        tile = 3  # the wider tile the engine may take here gives the same bits
    ref = states(c, prec, tile, 4)
    got = states(c, prec, None, 0)
    for a, b in zip(ref, got):
        assert np.isfinite(a).all()
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", FORMS)
@pytest.mark.parametrize("n", [(21, 21, 2), (40, 33, 7), (300, 200, 3)])
def test_2d_planes_evolve_independently(n, prec):
    c = smooth([n], 2, 5, reconstruct=abi.RECON_MUSCL, flux_split=abi.FLUX_ROE, compat=abi.COMPAT_REFERENCE)
    c.cfg.update(timestep_set=abi.DT_FIXED, dt=1e-3)
    whole = states(c, prec, None, 0)[0]
    for k in range(n[2]):
        one = smooth([(n[0], n[1], 1)], 2, 5, reconstruct=abi.RECON_MUSCL, flux_split=abi.FLUX_ROE)
        one.cfg.update(timestep_set=abi.DT_FIXED, dt=1e-3)
        one.states[0] = c.states[0][:, k:k + 1].copy()
        assert np.array_equal(states(one, prec, None, 0)[0][:, 0], whole[:, k])


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_FP32_FLUX])
def test_batch_shares_the_ctas(prec):
    members = [smooth([s], 3, 20 + i, reconstruct=abi.RECON_MUSCL, flux_split=abi.FLUX_ROE, precision=prec)
               for i, s in enumerate([(40, 24, 30), (16, 16, 64), (70, 9, 3), (24, 50, 18)])]
    s = Solver(members[0].config())
    s.remove_case(0)
    ids = []
    for c in members:
        c.apply(s, case_id=s.add_case(c.config()))
        ids.append(c.block_ids[0])
    s.step(3)
    for c, b in zip(members, ids):
        assert np.array_equal(s.get_state(b), states(c, prec, None, 0, steps=3)[0])
    s.close()
