"""The contour chain applied one axis at a time (csrc/axis_conv.cuh): every line
length on every axis, uneven boxes, both groupings of the y and z lines and
every tile width, against 3-D transforms in FP64 numpy.

Tolerances: a step is six 1-D transforms of n <= 128 points a value, each with
an error of a few eps log2(n); over N <= 6 steps that stays below 200 eps
relative to the largest value: 5e-14 in FP64, 2.4e-5 in FP32 (whose stated
phi tolerance is 1e-5)."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FP64_TOL, FP32_TOL = 5e-14, 1e-5
LENGTHS = (8, 12, 16, 20, 24, 32, 40, 48, 64, 80, 96, 128)
PAIRS = tuple((n, n) for n in LENGTHS) + ((12, 20), (24, 16), (16, 32), (32, 64))
# every length along x, every (my, mz) pair, small and large against each other
MESHES = tuple((LENGTHS[-1 - i] if n * n < 2500 else LENGTHS[i % 6], n, n) for i, n in enumerate(LENGTHS)) + \
    tuple((nx, ny, nz) for nx, (ny, nz) in zip((64, 96, 40, 12), PAIRS[-4:])) + ((128, 8, 8), (8, 128, 128))


@pytest.fixture(scope="module")
def lfts(native_lib):
    import lfts_cpu_b200
    return lfts_cpu_b200


def weights(m, L, N):
    k = [np.fft.fftfreq(n, 1.0 / n) / l for n, l in zip(m, L)]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + (k[2] ** 2)[None, None, : m[2] // 2 + 1]
    return np.exp(-4.0 * np.pi ** 2 * k2 / (6.0 * N))


def conv(q, g):
    return np.fft.irfftn(g * np.fft.rfftn(q), s=q.shape, axes=(0, 1, 2))


def box(m):
    return tuple(n / d for n, d in zip(m, (16.0, 15.0, 17.0)))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("m", MESHES)
def test_chain_of_every_length(lfts, m, precision):
    N, NA = 5, 2
    L, M = box(m), int(np.prod(m))
    w = np.random.default_rng(M).normal(0.0, 1.0, 2 * M)
    s = lfts.System(N, NA, 15.0, 50.0, 0.5, m, L, precision=precision)
    s.set_fields(w)
    g = weights(m, L, N)
    hA, hB = (np.exp(-x / N).reshape(m) for x in (w[:M] + w[M:], w[M:] - w[:M]))
    q, qd = [hA], [hB]
    for i in range(1, N):
        q.append((hA if i < NA else hB) * conv(q[-1], g))
        qd.append((hB if i < N - NA else hA) * conv(qd[-1], g))
    tol = FP64_TOL if precision == 0 else FP32_TOL
    first = None
    for cw in (8, 16, 32):
        t = dict(s.tiles(), pencil_cw=cw, phi_in_chain=0)
        s.set_tiles(**t)
        lnq = s.calc_concs()
        p = s.propagators()
        assert abs(lnq - np.log(q[-1].mean())) < tol * max(1.0, abs(lnq))
        for i in range(1, N + 1):
            assert rel_err(p[i, 0], q[i - 1].ravel()) < tol, (cw, i)
            assert rel_err(p[i, 1], qd[i - 1].ravel()) < tol, (cw, i)
        if first is None:
            first = (lnq, p)
        assert lnq == first[0] and np.array_equal(p, first[1]), cw  # the tiles change no value
    s.close()


@pytest.mark.parametrize("m", [(16, 16, 16), (24, 12, 20), (64, 64, 64), (128, 32, 64)])
def test_noalloc_step_on_8_byte_aligned_arrays(native_lib, m):
    """The caller's arrays need no more than a double's alignment, and one
    chain's non-finite values stay out of the other."""
    import torch

    from lfts_cpu_b200.capi import Params
    N, NA, M, L = 7, 3, int(np.prod(m)), box(m)
    p = Params()
    p.N, p.NA, p.XbN, p.C, p.dt = N, NA, 15.0, 50.0, 0.5
    for d in range(3):
        p.m[d], p.L[d] = m[d], L[d]
    rng = np.random.default_rng(M)
    q, h = rng.uniform(0.2, 1.5, 2 * M), rng.uniform(0.5, 1.2, 2 * M)
    g = weights(m, L, N)
    buf = torch.zeros(3, 2 * M + 1, dtype=torch.float64, device="cuda")
    qd, hd, od = (b[1:] for b in buf)  # 8 bytes past a 16-byte boundary
    if any(t.data_ptr() % 16 == 0 for t in (qd, hd, od)):
        qd, hd, od = (torch.zeros(2 * M + 1, dtype=torch.float64, device="cuda")[1:] for _ in range(3))
    assert qd.data_ptr() % 16 == 8 and hd.data_ptr() % 16 == 8 and od.data_ptr() % 16 == 8
    for bad in (None, 1, 0):
        qb = q.copy()
        if bad is not None:
            qb[bad * M + 3] = np.nan
        qd.copy_(torch.from_numpy(qb))
        hd.copy_(torch.from_numpy(h))
        torch.cuda.synchronize()
        for i in (2, 5):
            rc = native_lib.lfts_step_fwd_noalloc(C.byref(p), C.c_void_p(qd.data_ptr()), C.c_void_p(od.data_ptr()),
                                                  C.c_void_p(hd.data_ptr()), i, None)
            assert rc == 0
            torch.cuda.synchronize()
            got = od.cpu().numpy()
            hs = (0 if i < NA else 1, 1 if i < N - NA else 0)
            for c in (0, 1):
                if c == bad:
                    assert np.all(np.isnan(got[c * M:(c + 1) * M]))
                    continue
                ref = conv(q[c * M:(c + 1) * M].reshape(m), g).ravel() * h[hs[c] * M:(hs[c] + 1) * M]
                assert rel_err(got[c * M:(c + 1) * M], ref) < FP64_TOL


def test_noalloc_step_in_a_captured_graph(native_lib):
    """After a first call, the step can be captured into a graph and replayed on
    new contents of the same arrays."""
    import torch

    from lfts_cpu_b200.capi import Params
    m, N, NA = (16, 32, 64), 7, 3
    M, L = int(np.prod(m)), box((16, 32, 64))
    p = Params()
    p.N, p.NA, p.XbN, p.C, p.dt = N, NA, 15.0, 50.0, 0.5
    for d in range(3):
        p.m[d], p.L[d] = m[d], L[d]
    q, h, out = (torch.ones(2 * M, dtype=torch.float64, device="cuda") for _ in range(3))

    def call():
        st = torch.cuda.current_stream().cuda_stream
        assert native_lib.lfts_step_fwd_noalloc(C.byref(p), C.c_void_p(q.data_ptr()), C.c_void_p(out.data_ptr()),
                                                C.c_void_p(h.data_ptr()), 2, C.c_void_p(st)) == 0

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for seed in (1, 2):
        rng = np.random.default_rng(seed)
        qh, hh = rng.uniform(0.2, 1.5, 2 * M), rng.uniform(0.5, 1.2, 2 * M)
        q.copy_(torch.from_numpy(qh))
        h.copy_(torch.from_numpy(hh))
        graph.replay()
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        g = weights(m, L, N)
        for c, half in ((0, 0), (1, 1)):  # step 2 of NA = 3, NB = 4
            ref = conv(qh[c * M:(c + 1) * M].reshape(m), g).ravel() * hh[half * M:(half + 1) * M]
            assert rel_err(got[c * M:(c + 1) * M], ref) < FP64_TOL


@pytest.mark.parametrize("m", [(128, 12, 12), (96, 12, 20), (64, 20, 20), (48, 24, 16), (80, 16, 32), (40, 40, 40),
                               (12, 32, 64), (20, 48, 48), (64, 64, 64), (32, 80, 80), (24, 96, 96), (8, 128, 128)])
def test_fp32_chain_of_a_default_context(lfts, m, monkeypatch):
    """FP32-mixed contexts above 16384 points run this chain until set_tiles is called."""
    N, NA = 5, 2
    L, M = box(m), int(np.prod(m))
    w = np.random.default_rng(M).normal(0.0, 1.0, 2 * M)
    g = weights(m, L, N)
    hA, hB = (np.exp(-x / N).reshape(m) for x in (w[:M] + w[M:], w[M:] - w[:M]))
    q = [hA]
    for i in range(1, N):
        q.append((hA if i < NA else hB) * conv(q[-1], g))
    monkeypatch.setenv("LFTS_AUTOTUNE", "0")
    monkeypatch.setenv("LFTS_PHI_IN_CHAIN", "0")
    first = None
    for cw in (8, 16, 32):
        monkeypatch.setenv("LFTS_PENCIL_CW", str(cw))
        s = lfts.System(N, NA, 15.0, 50.0, 0.5, m, L, precision=1)
        assert s.tiles()["pencil_cw"] == cw
        s.set_fields(w)
        lnq, p = s.calc_concs(), s.propagators()
        s.close()
        assert abs(lnq - np.log(q[-1].mean())) < FP32_TOL * max(1.0, abs(lnq))
        for i in range(1, N + 1):
            assert rel_err(p[i, 0], q[i - 1].ravel()) < FP32_TOL, (cw, i)
        first = first or (lnq, p)
        assert lnq == first[0] and np.array_equal(p, first[1]), cw
