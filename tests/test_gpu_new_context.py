"""A new context and a new replica hold no concentrations yet, whether their tiles were
timed at their creation or taken from an earlier one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,m,N", [(0, (24, 12, 20), 5), (1, (24, 12, 20), 5), (1, (64, 32, 64), 9),
                                           (1, (96, 96, 96), 6)])
def test_new_contexts_are_alike(native_lib, precision, m, N):
    import lfts_cpu_b200 as lfts
    w = np.random.default_rng(1).normal(0.0, 0.5, 2 * int(np.prod(m)))
    for _ in range(2):
        s = lfts.System(N, 2, 15.0, 50.0, 0.5, m, (4.0, 4.0, 4.0), precision=precision)
        s.set_fields(w)
        f = s.get_fields()
        s.close()
        assert np.array_equal(f[:w.size], w) and not f[w.size:].any()


def test_new_replicas_are_alike(native_lib):
    import lfts_cpu_b200 as lfts
    reps = [{"N": 5, "NA": 2, "XbN": 15.0, "C": 50.0, "dt": 0.5, "m": (n, n, n), "L": (3.0, 3.0, 3.0), "seed": n}
            for n in (16, 24, 16)]
    for _ in range(2):
        e = lfts.Ensemble(reps)
        for r, d in enumerate(reps):
            w = np.full(2 * d["m"][0] ** 3, 0.25)
            e.set_fields(r, w)
            f = e.get_fields(r)
            assert np.array_equal(f[:w.size], w) and not f[w.size:].any()
        e.close()
