"""The concentration pass over the stored propagators: the sum over the monomers
split over 1 to 32 threads a mesh vector (csrc/field_kernels.cuh, conc_slices)
gives phi of the stored slots, at the chain lengths where the split changes.

A sum of N <= 65 products in FP64 is off by at most N eps = 7e-15 of its terms,
all positive; phi- is the difference of two such sums, so errors are relative to
phi+: 2e-14."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("m", [(8, 12, 20), (16, 16, 16), (20, 40, 40), (48, 48, 48), (64, 64, 64)])
def test_phi_of_the_stored_slots(native_lib, m, precision):
    import lfts_cpu_b200 as lfts
    M = int(np.prod(m))
    w = np.random.default_rng(M).normal(0.0, 1.0, 2 * M)
    for N, NA in ((2, 1), (3, 3), (7, 2), (8, 0), (15, 9), (16, 8), (31, 11), (65, 20)):
        s = lfts.System(N, NA, 15.0, 50.0, 0.5, m, tuple(n / 16.0 for n in m), precision=precision)
        s.set_fields(w)
        s.set_tiles(**dict(s.tiles(), phi_in_chain=0))
        lnq = s.calc_concs()
        phi = s.get_fields()[2 * M:]
        p = s.propagators()
        s.close()
        # slot i = (q_i, q^_{N+1-i}); hA = q_1's and hB = q^_N's factor: slot 1
        prod = [p[i, 0] * p[N + 1 - i, 1] for i in range(1, N + 1)]
        A = sum(prod[:NA], np.zeros(M)) / (N * np.exp(lnq) * p[1, 0])
        B = sum(prod[NA:], np.zeros(M)) / (N * np.exp(lnq) * p[1, 1])
        scale = np.max(np.abs(A + B))
        assert np.max(np.abs(phi[:M] - (A - B))) < 2e-14 * scale, (N, NA)
        assert np.max(np.abs(phi[M:] - (A + B))) < 2e-14 * scale, (N, NA)
