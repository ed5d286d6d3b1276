"""Residual norms and the CFL time step of the finalize kernel against the
oracle, over the ways its eight warps share a case's blocks: several warps per
block, one each, more blocks than warps, fewer tasks than lanes and more than
one round of loads per lane."""
import numpy as np
import pytest

import oracle as orc
from fvm3d import abi, cases
from fvm3d.solver import Solver

pytestmark = pytest.mark.gpu

# The oracle adds the n squared values of a block one after the other: its sum
# of positive terms is within n / 2 ulp at worst and about sqrt(n) / 2 ulp as
# a rule (n = 590,000 cells: 400 ulp, 9e-14); the kernel's tree is far closer.
RTOL = 1e-12


def run(blocks, steps=2, **cfg):
    base = dict(idimension=2, reconstruct=abi.RECON_MUSCL, limiter=abi.LIMITER_MINMOD, kappa=1.0 / 3.0,
                flux_split=abi.FLUX_ROE, entropy_fix=0.2, rk_stages=3, timestep_set=abi.DT_CFL, cfl=0.4)
    base.update(cfg)
    c = cases.Case(name="finalize", cfg=base)
    rng = np.random.default_rng(len(blocks) * 1000 + blocks[0][0])
    for n in blocks:
        c.blocks.append((n, (0.1, 0.1, 0.1)))
        sh = (n[2], n[1], n[0])
        f = lambda a, b: rng.uniform(a, b, sh)  # noqa: E731
        c.states.append(cases.prim_to_cons(f(0.8, 1.2), f(-0.2, 0.2), f(-0.2, 0.2), f(-0.2, 0.2), f(0.8, 1.2)))
        c.origins.append((0, 0, 0))
    g = c.apply(Solver(c.config()))
    o = c.apply(orc.Oracle(c.config()))
    tg, rg, lg = g.step(steps)
    to, ro, lo, _ = o.step(steps)
    assert tg == to
    np.testing.assert_allclose(rg, ro, rtol=RTOL, atol=0)
    np.testing.assert_allclose(lg, lo, rtol=2 * RTOL, atol=0)
    for b in range(len(blocks)):
        assert np.array_equal(g.get_state(b), o.get_state(b))


@pytest.mark.parametrize("nblocks", [1, 2, 3, 4, 5, 7, 8, 9, 17])
def test_blocks_share_warps(nblocks):
    run([(9 + b, 7, 1 + b % 2) for b in range(nblocks)])


@pytest.mark.parametrize("n", [(1, 1, 1), (300, 300, 1), (40, 30, 1)])
def test_task_counts(n):
    run([n])


def test_many_tasks_of_one_block():
    # 64 x 36 tiles of 32 x 8: more than 8 warps x 32 lanes x 8 loads
    run([(2048, 288, 1)], steps=1)
