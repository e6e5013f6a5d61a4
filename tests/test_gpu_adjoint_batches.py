"""Gradients of H with the adjoint's terms launched several at a time and its
checkpointed segments recomputed two at a time: every remainder of either, against
numpy in FP64 (dQ/dL_a from the spectra of q_i and q^_{i+1}; dH/dL = -dQ/dL / Q).

The terms' sum is of N M products of spectra; the tests of the FP64 path hold it to
1e-10 of its largest component."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def exact_dL(w, m, L, N, NA):
    M = int(np.prod(m))
    hA, hB = (np.exp(-x / N).reshape(m) for x in (w[:M] + w[M:], w[M:] - w[:M]))
    k = [np.fft.fftfreq(n, 1.0 / n) for n in m]
    k[2] = np.arange(m[2] // 2 + 1.0)
    ks = [k[d].reshape([-1 if e == d else 1 for e in range(3)]) for d in range(3)]
    g = np.exp(-4.0 * np.pi ** 2 * sum((ks[d] / L[d]) ** 2 for d in range(3)) / (6.0 * N))
    conv = lambda t: np.fft.irfftn(g * np.fft.rfftn(t), s=m, axes=(0, 1, 2))  # noqa: E731
    q, qd = [hA], [hB]
    for i in range(1, N):
        q.append((hA if i < NA else hB) * conv(q[-1]))
        qd.append((hB if i < N - NA else hA) * conv(qd[-1]))
    wt = np.full(m[2] // 2 + 1, 2.0)
    wt[0] = wt[-1] = 1.0
    acc = sum((np.fft.rfftn(q[i - 1]) * np.conj(np.fft.rfftn(qd[N - i - 1]))).real for i in range(1, N))
    Q = q[-1].mean()
    c = 4.0 * np.pi ** 2 / (3.0 * N)
    return np.array([-(c * ks[d] ** 2 / L[d] ** 3 * g * wt * acc).sum() / M / M / Q for d in range(3)])


@pytest.mark.parametrize("m", [(12, 24, 16), (16, 16, 16), (24, 64, 64)])
@pytest.mark.parametrize("N,NA", [(2, 1), (3, 3), (6, 0), (17, 5), (18, 9), (40, 13)])
def test_batches_and_segments(native_lib, m, N, NA):
    import lfts_cpu_b200 as lfts
    M, L = int(np.prod(m)), tuple(n / d for n, d in zip(m, (9.0, 8.0, 10.0)))
    w = np.random.default_rng(N).normal(0.0, 1.5, 2 * M)
    ref = exact_dL(w, m, L, N, NA)
    s = lfts.System(N, NA, 15.0, 50.0, 0.5, m, L)
    s.set_fields(w)
    for every in (0, 1, 2, 3, 5, 16, N - 1, N, 1000):
        dL, _, _ = s.backward(every)
        assert np.max(np.abs(dL - ref)) < 1e-10 * np.max(np.abs(ref)), every
    s.close()
