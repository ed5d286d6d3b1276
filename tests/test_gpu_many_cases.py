"""Case states of an engine with more cases than one small copy brings back:
the states of the last ones come in a copy of their own, beside the error flag."""
import numpy as np
import pytest

from fvm3d import abi, cases
from fvm3d.solver import Solver

pytestmark = pytest.mark.gpu

CFG = dict(idimension=2, reconstruct=abi.RECON_MUSCL, limiter=abi.LIMITER_MINMOD, kappa=1.0 / 3.0,
           flux_split=abi.FLUX_ROE, entropy_fix=0.2, rk_stages=3, timestep_set=abi.DT_CFL, cfl=0.4)
N = (9, 7, 1)


def state(i):
    rng = np.random.default_rng(i)
    f = lambda a, b: rng.uniform(a, b, (1, N[1], N[0]))  # noqa: E731
    return cases.prim_to_cons(f(0.8, 1.2), f(-0.2, 0.2), f(-0.2, 0.2), f(-0.2, 0.2), f(0.8, 1.2))


def test_states_of_late_case_ids():
    s = Solver(**CFG)
    ids = [0] + [s.add_case(abi.make_config(**CFG)) for _ in range(219)]
    for i, cid in enumerate(ids):
        b = s.add_block(N, (0.1, 0.1, 0.1)) if cid == 0 else s.add_case_block(cid, N, (0.1, 0.1, 0.1))
        s.set_state(b, state(i))
    s.step(2)
    for i in (0, 1, 60, 80, 88, 89, 90, 91, 92, 100, 150, 219):
        one = Solver(**CFG)
        one.add_block(N, (0.1, 0.1, 0.1))
        one.set_state(0, state(i))
        one.step(2)
        a, b = s.case_state(ids[i]), one.case_state(0)
        assert a["step"] == 2 and a["status"] == 0
        for k in ("t", "dt", "step", "status"):
            assert a[k] == b[k], (i, k)
        assert np.array_equal(a["res_abs"], b["res_abs"]) and np.array_equal(a["res_rel"], b["res_rel"])
        one.close()
    s.close()
