"""The allocation-free readback takes time in proportion to its particles up to
the largest id space: twice the particles, at most twice the time (and a tenth
for the clock).  A scan of all words by one CTA took three times as long."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def microseconds(n):
    from flipengine3d_gb300.fluidsimulation import order_particles_by_id_noalloc
    rng = np.random.default_rng(n)
    ids = [torch.from_numpy(rng.permutation(n).astype(np.int32)).cuda() for _ in range(3)]
    xyz, out = torch.rand(3, n, device="cuda"), torch.empty(n, 3, device="cuda")
    p, stream = xyz.data_ptr(), torch.cuda.current_stream().cuda_stream
    best = np.inf
    for rep in range(12):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for q in range(9):
            order_particles_by_id_noalloc(p, p + 4 * n, p + 8 * n, ids[q % 3].data_ptr(), n, n, out.data_ptr(), stream)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1000 / 9)
    assert torch.equal(out, xyz.t()[torch.argsort(ids[8 % 3].long())])
    return best


@pytest.mark.gpu
def test_time_grows_with_the_particles(gpu):
    half, full = microseconds(1 << 19), microseconds(1 << 20)
    assert full <= 2.2 * half, (half, full)
