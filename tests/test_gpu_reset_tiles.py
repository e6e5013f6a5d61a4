"""lfts_reset_tiles takes a context back to the chain and tiles it was created with:
set_tiles on an FP32-mixed context selects the chain by 3-D transforms, tiles that
get_tiles reported included, and the way back gives the first results bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def results(s, w):
    s.set_fields(w)
    lnq = s.calc_concs()
    phi, p = s.get_fields()[w.size:], s.propagators()
    try:
        s.mix(6, 1e-12)
    except RuntimeError:
        pass
    return lnq, phi, p, s.get_fields()


@pytest.mark.parametrize("device_loop", [False, True])
@pytest.mark.parametrize("precision,m,default", [(0, (32, 32, 32), False), (1, (32, 32, 32), True),
                                                 (1, (20, 20, 20), True), (1, (64, 64, 64), False),
                                                 (1, (40, 32, 64), False), (1, (96, 96, 96), False)])
def test_back_to_the_created_chain(native_lib, monkeypatch, precision, m, default, device_loop):
    import lfts_cpu_b200 as lfts
    monkeypatch.setenv("LFTS_DEVICE_MIX", "1" if device_loop else "0")
    w = np.random.default_rng(5).normal(0.0, 0.6, 2 * int(np.prod(m)))
    s = lfts.System(7, 3, 16.0, 100.0, 0.5, m, tuple(x / 16.0 for x in m), precision=precision)
    assert s.by_transforms is default
    t, first = s.tiles(), results(s, w)
    s.set_tiles(**t)
    assert s.by_transforms is (precision == 1)
    results(s, w)
    s.reset_tiles()
    assert s.by_transforms is default and s.tiles() == t
    for a, b in zip(results(s, w), first):
        assert np.array_equal(a, b)
    s.close()
