"""The autotuner's search, with the library calls replaced: it times every
combination that differs once, and keeps none that has no effect."""
import types

import pytest

from fvm3d import tuning


@pytest.mark.parametrize("idim,expected", [(3, 4 * (1 + 4 * 4)), (2, 4)])
def test_search_times_each_configuration_once(monkeypatch, idim, expected):
    timed, now = [], {}
    monkeypatch.setattr(tuning, "set_tuning", lambda s, c, t, z: now.update(tile=t, z=z))
    monkeypatch.setattr(tuning, "set_tail_split", lambda s, c, sp: now.update(split=sp))

    def time_step(s, reps):
        if reps > 1:
            timed.append((now["tile"], now["z"], now["split"]))
        # a later repetition of the same configuration looks faster, as noise would have it
        return 1.0 - 1e-6 * len(timed) + (0.0 if now["z"] == 0 else 1.0)

    monkeypatch.setattr(tuning, "time_step", time_step)
    cfg = types.SimpleNamespace(idimension=idim, reconstruct=202, flux_split=303, compat=0, precision=1)
    best = tuning.autotune(types.SimpleNamespace(cfg=cfg), 1000, use_cache=False)
    # the tail split acts on chunked tasks only: with z chunk 0 the engine splits evenly by itself
    effective = [(t, z, sp if z > 0 else 1) for t, z, sp in timed]
    assert len(timed) == len(set(effective)) == expected
    assert best[1] == 0 and best[3] == 1
    assert (now["tile"], now["z"], now["split"]) == (best[0], 0, 1)
