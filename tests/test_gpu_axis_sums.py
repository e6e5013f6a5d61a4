"""The axis-by-axis FP32-mixed chain as a context runs it by default, without
set_tiles (which selects the chain by 3-D transforms): its concentration sums in the
chain and in the separate pass, both of its chains, chain lengths that end along x
(even N) and along y and z (odd N), and the device-side Anderson loop.

Tolerances are those of the FP32-mixed path: 1e-5 of the largest value, for ln Q of
max(1, |ln Q|).  ln Q and the propagators do not depend on where the sums are formed."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FP32_TOL = 1e-5


def box(m):
    return tuple(n / d for n, d in zip(m, (16.0, 15.0, 17.0)))


def default_context(monkeypatch, N, NA, m, phi, device_loop=False):
    import lfts_cpu_b200 as lfts
    with monkeypatch.context() as mp:
        mp.setenv("LFTS_AUTOTUNE", "0")
        mp.setenv("LFTS_PHI_IN_CHAIN", str(phi))
        mp.setenv("LFTS_DEVICE_MIX", "1" if device_loop else "0")
        s = lfts.System(N, NA, 16.0, 100.0, 0.5, m, box(m), precision=1)
    assert not s.by_transforms and s.tiles()["phi_in_chain"] == phi
    return s


@pytest.mark.parametrize("m,N,NA", [
    ((96, 96, 96), 2, 1), ((96, 96, 96), 3, 2), ((96, 96, 96), 7, 3), ((96, 96, 96), 8, 8), ((96, 96, 96), 8, 0),
    ((128, 128, 128), 2, 1), ((128, 128, 128), 3, 1), ((128, 128, 128), 8, 5), ((128, 128, 128), 64, 25),
    ((96, 128, 128), 7, 7), ((128, 96, 96), 6, 0), ((128, 96, 96), 5, 4)])
def test_sums_in_the_chain_and_apart(native_lib, monkeypatch, m, N, NA):
    import lfts_cpu_b200 as lfts
    M = int(np.prod(m))
    w = np.random.default_rng(N * 100 + NA).normal(0.0, 0.5, 2 * M)
    out = []
    for phi in (0, 1):
        s = default_context(monkeypatch, N, NA, m, phi)
        s.set_fields(w)
        out.append((s.calc_concs(), s.get_fields()[2 * M:], s.propagators() if N <= 8 else None))
        s.close()
    (lnq0, phi0, p0), (lnq1, phi1, p1) = out
    assert lnq1 == lnq0 and (p0 is None or np.array_equal(p1, p0))
    s = lfts.System(N, NA, 16.0, 100.0, 0.5, m, box(m))
    s.set_fields(w)
    lnq64 = s.calc_concs()
    phi64 = s.get_fields()[2 * M:]
    p64 = s.propagators() if N <= 8 else None
    s.close()
    assert abs(lnq0 - lnq64) < FP32_TOL * max(1.0, abs(lnq64))
    assert rel_err(phi0, phi64) < FP32_TOL and rel_err(phi1, phi64) < FP32_TOL
    if p64 is not None:
        for i in range(1, N + 1):
            for chain in (0, 1):
                assert rel_err(p0[i, chain], p64[i, chain]) < FP32_TOL, (i, chain)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("N,NA", [(2, 1), (4, 1), (5, 2)])
@pytest.mark.parametrize("m", [(128, 12, 12), (96, 24, 16), (48, 24, 16), (80, 16, 32), (40, 40, 40), (12, 32, 64),
                               (20, 48, 48), (64, 64, 64), (32, 80, 80), (24, 96, 96), (8, 128, 128)])
def test_both_chains_of_a_default_context(native_lib, m, N, NA, precision):
    """Against 3-D transforms in FP64 numpy."""
    import lfts_cpu_b200 as lfts
    M, L = int(np.prod(m)), box(m)
    w = np.random.default_rng(M + N).normal(0.0, 1.0, 2 * M)
    k2 = sum((np.fft.fftfreq(n, 1.0 / n) / l).reshape([-1 if a == d else 1 for a in range(3)]) ** 2
             for d, (n, l) in enumerate(zip(m, L)))
    g = np.exp(-4.0 * np.pi ** 2 * k2 / (6.0 * N))
    hA, hB = (np.exp(-x / N).reshape(m) for x in (w[:M] + w[M:], w[M:] - w[:M]))
    q, qd = [hA], [hB]
    for i in range(1, N):
        q.append((hA if i < NA else hB) * np.fft.ifftn(g * np.fft.fftn(q[-1])).real)
        qd.append((hB if i < N - NA else hA) * np.fft.ifftn(g * np.fft.fftn(qd[-1])).real)
    s = lfts.System(N, NA, 16.0, 100.0, 0.5, m, L, precision=precision)
    assert not s.by_transforms
    s.set_fields(w)
    lnq, p = s.calc_concs(), s.propagators()
    s.close()
    tol = FP32_TOL if precision else 5e-14
    assert abs(lnq - np.log(q[-1].mean())) < tol * max(1.0, abs(lnq))
    assert abs(lnq - np.log(qd[-1].mean())) < tol * max(1.0, abs(lnq))
    for i in range(1, N + 1):
        assert rel_err(p[i, 0], q[i - 1].ravel()) < tol, i
        assert rel_err(p[i, 1], qd[i - 1].ravel()) < tol, i


def mix(s):
    import lfts_cpu_b200 as lfts
    try:
        return s.mix()
    except lfts.LftsError as e:  # the pure-A system's mixing diverges, in FP64 too
        return str(e)


@pytest.mark.parametrize("m,N,NA,phi", [((96, 96, 96), 8, 3, 1), ((96, 96, 96), 7, 4, 0), ((128, 128, 128), 7, 3, 1),
                                        ((64, 64, 64), 9, 4, 0), ((40, 16, 32), 8, 8, 0)])
def test_device_loop_on_a_default_context(native_lib, monkeypatch, m, N, NA, phi):
    """The same counts, fields and outcome as the loop on the host."""
    M = int(np.prod(m))
    w = np.random.default_rng(M + N).normal(0.0, 0.6, 2 * M)
    noise = np.random.default_rng(1).normal(0.0, 2.0, (2, M))
    out = []
    for device_loop in (False, True):
        s = default_context(monkeypatch, N, NA, m, phi, device_loop)
        s.set_fields(w)
        ks = [mix(s)]
        s.calc_concs()
        s.langevin_init(noise[0])
        s.langevin_step(noise[1])
        ks.append(mix(s))
        s.calc_concs()
        out.append((ks, s.get_fields(), s.anderson_stats()))
        s.close()
    assert out[0][0] == out[1][0] and out[0][2] == out[1][2]
    assert all(isinstance(k, int) for k in out[0][0]) == (NA < N)
    assert np.array_equal(out[0][1], out[1][1], equal_nan=True)
