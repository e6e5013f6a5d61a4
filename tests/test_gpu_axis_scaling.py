"""FP32-mixed propagators near the small end of single precision: w+ shifted by a
constant scales q_i by exp(-shift i / N) and changes no concentration.  At a shift of 86
q_N is of the size of 4e-38, 3 times the smallest normal number, and the chain has to hold
its values at that size between the axes too: the propagators keep the FP32-mixed
tolerance, 1e-5 of the largest value, which the transform chain holds there as well."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FP32_TOL = 1e-5


@pytest.mark.parametrize("m", [(128, 128, 128), (64, 64, 64), (96, 80, 80), (128, 32, 64)])
def test_fp32_propagators_of_shifted_fields(native_lib, m):
    import lfts_cpu_b200 as lfts
    N, NA, M = 32, 12, int(np.prod(m))
    w = np.random.default_rng(1).normal(0.0, 0.7, 2 * M)
    w[M:] += 86.0
    out = []
    for precision in (0, 1):
        s = lfts.System(N, NA, 16.0, 100.0, 0.5, m, tuple(x / 16.0 for x in m), precision=precision)
        s.set_fields(w)
        lnq = s.calc_concs()
        p = s.propagators()
        out.append((lnq, s.get_fields()[2 * M:], p[[N - 4, N]].copy()))
        s.close()
    (lnq64, phi64, q64), (lnq32, phi32, q32) = out
    assert abs(lnq32 - lnq64) < FP32_TOL
    assert rel_err(phi32, phi64) < FP32_TOL
    for i in (0, 1):
        for chain in (0, 1):
            assert rel_err(q32[i, chain], q64[i, chain]) < FP32_TOL, (i, chain)
