"""The allocation-free readback at the sizes where its words and its one-CTA scan
change over: less than a word of ids, whole words and one id more or less, a
word a thread of the scan and one more, the largest id space, every id present.
Against NumPy's stable order by id, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("space,n", [(1, 1), (31, 9), (32, 32), (33, 1), (1000, 640), (32767, 20000), (32768, 32768),
                                     (32769, 32000), (65537, 65000), (1 << 20, 700001), (1 << 20, 1 << 20)])
def test_order_at_word_edges(gpu, space, n):
    from flipengine3d_gb300.fluidsimulation import order_particles_by_id_noalloc
    rng = np.random.default_rng(space + n)
    ids = rng.permutation(space)[:n].astype(np.int32)
    xyz = rng.random((3, n), dtype=np.float32)
    d_ids, d_xyz = torch.from_numpy(ids).cuda(), torch.from_numpy(xyz).cuda()
    out = torch.full((n, 3), -1.0, dtype=torch.float32, device="cuda")
    step = 4 * n
    for _ in range(2):   # the second call finds the first one's scratch
        order_particles_by_id_noalloc(d_xyz.data_ptr(), d_xyz.data_ptr() + step, d_xyz.data_ptr() + 2 * step, d_ids.data_ptr(),
                                      n, space, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(out.cpu().numpy(), xyz.T[np.argsort(ids, kind="stable")])


@pytest.mark.gpu
def test_order_in_a_captured_graph(gpu):
    """The call captured into a graph and replayed with other particles in the same memory."""
    from flipengine3d_gb300.fluidsimulation import order_particles_by_id_noalloc
    n, space = 5000, 7001
    rng = np.random.default_rng(4)
    d_ids = torch.zeros(n, dtype=torch.int32, device="cuda")
    d_xyz = torch.zeros((3, n), dtype=torch.float32, device="cuda")
    out = torch.zeros((n, 3), dtype=torch.float32, device="cuda")

    def fill():
        ids, xyz = rng.permutation(space)[:n].astype(np.int32), rng.random((3, n), dtype=np.float32)
        d_ids.copy_(torch.from_numpy(ids))
        d_xyz.copy_(torch.from_numpy(xyz))
        return xyz.T[np.argsort(ids, kind="stable")]

    def call():
        p = d_xyz.data_ptr()
        order_particles_by_id_noalloc(p, p + 4 * n, p + 8 * n, d_ids.data_ptr(), n, space, out.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream)

    want = fill()
    call()   # loads the module
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for _ in range(3):
        want = fill()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
