"""What the FP64 update's tuner times is what the factorisation runs."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [250, 317])  # one outer block with columns behind it; a pair and 64 columns
def test_timed_updates_are_those_of_the_factorisation(n, monkeypatch, capfd):
    """At these sizes the timed steps are all the trailing updates there are, so the time of either candidate is
    the profiled sum of the factorisation's updates with that candidate, up to the gaps between launches (a tenth
    of these times) and the spread of a single timing."""
    from minigw_b200 import B200Backend
    from test_panel import _system

    sl = _system(n, n // 2, 4, 1900 + n)
    omegas = np.geomspace(1e-2, 50.0, 147)  # a geometry of its own: timed here, not in an earlier test
    with B200Backend(0) as be:
        be.load_slices(sl)
        monkeypatch.setenv("GWB200_VERBOSE", "1")
        be.screened_forms(omegas, sl.states)
        line = next(x for x in capfd.readouterr().err.splitlines() if "gwb200: update kernel" in x)
        monkeypatch.delenv("GWB200_VERBOSE")
        timed = dict(zip(("dmma", "ozaki"), (float(x) for x in re.findall(r"([0-9.]+) ms", line))))
        monkeypatch.setenv("GWB200_PROFILE", "1")
        for update in ("dmma", "ozaki"):
            monkeypatch.setenv("GWB200_FP64_UPDATE", update)
            run = min(be.screened_forms(omegas, sl.states)[1]["device_ms_update"] for _ in range(5))
            assert 0.8 < timed[update] / run < 1.25, (update, timed, run)
