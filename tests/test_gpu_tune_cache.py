"""The tuner's choices are kept for a process, each for the candidates that it was made
from: a variable that fixes a choice acts on every context and ensemble created under it,
also on a mesh that was tuned before with other values of it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,m,var,key,values", [
    (0, (24, 16, 32), "LFTS_PENCIL_CW", "pencil_cw", (8, 16, 32)),
    (1, (24, 16, 32), "LFTS_PENCIL_CW", "pencil_cw", (8, 16, 32)),
    (1, (96, 96, 96), "LFTS_PHI_IN_CHAIN", "phi_in_chain", (0, 1)),
    (0, (32, 32, 32), "LFTS_ONE_STREAM", "two_streams", (0, 1)),
])
def test_a_forced_choice_acts_on_every_context(native_lib, monkeypatch, precision, m, var, key, values):
    import lfts_cpu_b200 as lfts
    for v in values + values[::-1]:
        monkeypatch.setenv(var, str(v))
        s = lfts.System(6, 2, 15.0, 50.0, 0.5, m, (4.0, 4.0, 4.0), precision=precision)
        got = s.tiles()[key]
        s.close()
        assert got == (1 - v if key == "two_streams" else v)


def test_a_forced_choice_acts_on_every_ensemble(native_lib, monkeypatch):
    import lfts_cpu_b200 as lfts
    reps = [{"N": 6, "NA": 2, "XbN": 15.0, "C": 50.0, "dt": 0.5, "m": (24, 24, 24), "L": (3.0, 3.0, 3.0), "seed": r}
            for r in range(2)]
    for cw in (32, 16, 32):
        monkeypatch.setenv("LFTS_PENCIL_CW", str(cw))
        e = lfts.Ensemble(reps)
        got = e.tiles(0)["pencil_cw"]
        e.close()
        assert got == cw
