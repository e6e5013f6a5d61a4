"""LFTS_XH_CHAIN and LFTS_PLANE_SPLIT name a layout of the FP32-mixed chain by 3-D
transforms: a context created under them runs that chain with that layout, bit for bit
what lfts_set_tiles installs, and agrees with FP64 to the FP32-mixed tolerance.  Meshes
without the layout keep their chain."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FP32_TOL = 1e-5


def results(s, w):
    s.set_fields(w)
    return s.calc_concs(), s.get_fields()[w.size:], s.propagators()


@pytest.mark.parametrize("m,env,key,value", [
    ((128, 128, 128), {"LFTS_XH_CHAIN": "1"}, "h_in_pencil", 1),
    ((128, 128, 128), {"LFTS_XH_CHAIN": "0"}, "h_in_pencil", 0),
    ((96, 96, 96), {"LFTS_XH_CHAIN": "0"}, "h_in_pencil", 0),
    ((128, 128, 128), {"LFTS_PLANE_SPLIT": "8"}, "plane_split", 8),
    ((128, 128, 128), {"LFTS_PLANE_SPLIT": "8", "LFTS_AUTOTUNE": "0"}, "plane_split", 8),
    ((96, 128, 128), {"LFTS_XH_CHAIN": "1", "LFTS_PLANE_SPLIT": "1", "LFTS_AUTOTUNE": "0"}, "plane_split", 1),
])
@pytest.mark.parametrize("N,NA,phi", [(6, 2, "0"), (7, 7, "1")])
def test_layout_named_by_the_environment(native_lib, monkeypatch, m, env, key, value, N, NA, phi):
    import lfts_cpu_b200 as lfts
    w = np.random.default_rng(N).normal(0.0, 0.6, 2 * int(np.prod(m)))
    args = (N, NA, 16.0, 100.0, 0.5, m, tuple(x / 16.0 for x in m))
    with monkeypatch.context() as mp:
        mp.setenv("LFTS_PHI_IN_CHAIN", phi)
        for k, v in env.items():
            mp.setenv(k, v)
        s = lfts.System(*args, precision=1)
    t = s.tiles()
    assert t[key] == value
    got = results(s, w)
    s.close()
    s = lfts.System(*args, precision=1)
    s.set_tiles(**t)
    ref = results(s, w)
    s.close()
    assert got[0] == ref[0] and np.array_equal(got[1], ref[1]) and np.array_equal(got[2], ref[2])
    s = lfts.System(*args)
    lnq, phi64, p = results(s, w)
    s.close()
    assert abs(got[0] - lnq) < FP32_TOL * max(1.0, abs(lnq))
    assert rel_err(got[1], phi64) < FP32_TOL
    assert rel_err(got[2][:, 0], p[:, 0]) < FP32_TOL and rel_err(got[2][:, 1], p[:, 1]) < FP32_TOL


@pytest.mark.parametrize("m", [(64, 64, 64), (40, 40, 40)])
def test_meshes_without_the_layout_keep_their_chain(native_lib, monkeypatch, m):
    import lfts_cpu_b200 as lfts
    w = np.random.default_rng(1).normal(0.0, 0.6, 2 * int(np.prod(m)))
    out = []
    for env in ({}, {"LFTS_XH_CHAIN": "0"}, {"LFTS_PLANE_SPLIT": "8"}):
        with monkeypatch.context() as mp:
            for k, v in env.items():
                mp.setenv(k, v)
            s = lfts.System(6, 2, 16.0, 100.0, 0.5, m, tuple(x / 16.0 for x in m), precision=1)
        out.append(results(s, w))
        s.close()
    for r in out[1:]:
        assert r[0] == out[0][0] and np.array_equal(r[1], out[0][1]) and np.array_equal(r[2], out[0][2])
