"""The ends of CG solves: instances that end at different phases of a launch,
and solves that break down, over and over."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_instances_that_end_one_after_another(cuda):
    """A phase drains the tiles of an instance that ends at its start, beside the
    tiles of others; each instance keeps the bits of its own run every time."""
    import torch

    import shearwave_b200 as sw
    from shearwave_b200 import ops

    # more tiles than blocks, both tile shapes, limits one update apart
    shapes = [(40, 33, 70), (33, 34, 66), (21, 50, 33), (17, 19, 33)] * 5
    iters = [1 + k % 7 for k in range(len(shapes))]
    h = 0.5e-3
    rng = np.random.default_rng(11)
    f = [[torch.as_tensor(rng.standard_normal(s), device=cuda) for _ in range(3)] for s in shapes]
    alone = [sw.project_vector_field(*c, h, h, h, 1e-12, n) for c, n in zip(f, iters)]
    for _ in range(10):
        outs, stats = ops.project_batch([c[0] for c in f], [c[1] for c in f], [c[2] for c in f],
                                        [h] * 3 * len(f), [1e-12] * len(f), iters)
        for k, s in enumerate(shapes):
            both = outs[k].reshape(3, s[0], s[1], ops.pitch(s[2]))[..., :s[2]]
            assert all(torch.equal(a, b) for a, b in zip(alone[k], both)), k
            assert int(stats[k, 0]) == iters[k]


@pytest.mark.parametrize("shape", [(5, 6, 7), (17, 19, 33), (40, 33, 70)])
def test_breakdowns_end_the_launch(cuda, shape):
    """A negative modulus makes p.Ap negative: the first update phase finds it and the
    next phase ends the launch, every time, without a wait that runs out."""
    import torch

    import shearwave_b200 as sw

    g = torch.Generator(device="cuda").manual_seed(1)
    b = torch.randn(shape, device=cuda, dtype=torch.float64, generator=g)
    info = {}
    for _ in range(300):
        out = sw.elastic_solve_static(b, 0.5, 0.5, 0.5, -1.0, tol=1e-9, max_iters=50, info=info)
        assert info["iters"] == 0
    assert not bool(out.any())


def test_grids_one_after_another_in_one_workspace(cuda):
    """The tensor maps of a solve lie in its workspace: another grid's, at the same
    address, are not used for it."""
    import ctypes as C

    import torch

    import shearwave_b200 as sw
    from shearwave_b200 import _native, ops

    shapes = [(20, 30, 40), (30, 20, 40), (12, 50, 33), (40, 30, 20)]
    h = 0.5e-3
    g = torch.Generator(device="cuda").manual_seed(5)
    f = [[torch.randn(s, device=cuda, dtype=torch.float64, generator=g) for _ in range(3)]
         for s in shapes]
    ref = [sw.project_vector_field(*c, h, h, h, 1e-9, 30) for c in f]
    nb = max(int(_native.load().sw_project_workspace_bytes(*s)) for s in shapes)
    ws = torch.empty(nb, dtype=torch.uint8, device=cuda)
    for k in list(range(len(shapes))) * 25:
        nx, ny, nz = shapes[k]
        out = torch.empty((3, nx, ny, ops.pitch(nz)), dtype=torch.float64, device=cuda)
        st = _native.CGStats()
        _native.call("sw_project", _native.SW_F64, *(c.data_ptr() for c in f[k]), ny * nz, nz, 1,
                     nx, ny, nz, h, h, h, 1e-9, 30, out.data_ptr(), ws.data_ptr(), nb,
                     C.byref(st), torch.cuda.current_stream().cuda_stream)
        assert all(torch.equal(a, b) for a, b in zip(out[..., :nz], ref[k])), k
