"""Gradients of H on a device with little memory left: the scratch that batches the
adjoint's terms gives way to the checkpointed segment's rows, and without room for it
the terms go through the contour chain's own buffer.

At 128^3 a row of a recomputed segment takes 16 MiB and a term's spectra 33: storing all
propagators needs next to nothing beside the context, checkpoints every 4 steps need 4
rows.  The gradients are sums of the same terms in another order (1e-10 of the largest,
as for the FP64 path)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fill(leave):
    """Takes device memory until about `leave` MiB are free."""
    import torch
    hold = []
    torch.cuda.synchronize()
    while True:
        n = min(torch.cuda.mem_get_info()[0] - (leave << 20), 1 << 34) >> 21
        if n < 2:
            return hold
        hold.append(torch.empty(n << 21, dtype=torch.uint8, device="cuda"))


@pytest.mark.parametrize("every,leave", [(0, 16), (4, 96)])
def test_gradients_with_little_memory_left(native_lib, every, leave):
    import torch

    import lfts_cpu_b200 as lfts
    m, N = (128, 128, 128), 12
    s = lfts.System(N, 5, 16.0, 100.0, 0.5, m, (8.0, 8.0, 8.0))
    s.set_fields(np.random.default_rng(1).normal(0.0, 0.5, 2 * 128 ** 3))
    s.calc_concs()
    s.get_H()
    hold = fill(leave)
    try:
        tight = s.backward(every)
    finally:
        del hold
        torch.cuda.empty_cache()
    roomy = s.backward(every)
    s.close()
    assert np.max(np.abs(tight[0] - roomy[0])) < 1e-10 * np.max(np.abs(roomy[0]))
    assert tight[1:] == roomy[1:]
