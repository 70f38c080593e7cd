"""The CG solves at grids around the tiles and x chunks of their kernel.

Against the oracle's CG in float64.  Both sides stop at a relative residual
of 1e-12, so the projected forces differ by at most 2e-12 sqrt(lmax / lmin) of
the force's norm and the static solutions by 2e-12 lmax / lmin of theirs:
below 1e-9 and 1e-7 on these grids.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# both tile shapes (64 x 8 and 32 x 16), one cell past their edges, single
# planes, single rows, and chunks of one and of several planes along x
SHAPES = [(3, 3, 3), (4, 3, 5), (5, 17, 66), (9, 18, 34), (7, 10, 130), (40, 11, 65), (131, 5, 6),
          (6, 130, 35), (3, 9, 67), (17, 19, 33)]


def _rel(a, b):
    n = np.linalg.norm(b)
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / (n if n else 1.0))


@pytest.mark.parametrize("shape", SHAPES)
def test_projection_cg_at_tile_edges(cuda, shape):
    import shearwave_b200 as sw
    from oracle import shearwave_oracle as O

    rng = np.random.default_rng(sum(shape))
    h = (0.5e-3, 0.4e-3, 0.7e-3)
    f = [rng.standard_normal(shape) for _ in range(3)]
    ref = O.project_vector_field(*[c.copy() for c in f], *h, 1e-12, 3000, dtype=np.float64)
    out = sw.project_vector_field(*f, *h, 1e-12, 3000)
    norm = np.sqrt(sum(np.sum(c * c) for c in f))
    assert np.sqrt(sum(np.sum((a - b) ** 2) for a, b in zip(out, ref))) <= 1e-9 * norm


@pytest.mark.parametrize("field", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_static_solve_at_tile_edges(cuda, shape, field):
    import shearwave_b200 as sw
    from oracle import shearwave_oracle as O

    rng = np.random.default_rng(sum(shape) + 1)
    b = rng.standard_normal(shape)
    mu = 2.0 * (1 + 0.1 * rng.standard_normal(shape)) if field else 2.0
    h = (0.5, 0.4, 0.7)
    info = {}
    # a map makes the operator unsymmetric: compare a fixed number of updates
    tol, iters = (0.0, 5) if field else (1e-12, 3000)
    ref = O.elastic_solve_static(b, *h, mu, tol=tol, max_iters=iters, dtype=np.float64)
    out = sw.elastic_solve_static(b, *h, mu, tol=tol, max_iters=iters, info=info)
    assert _rel(out, ref) <= 1e-7, info


def test_batched_projection_with_ended_and_tiny_instances(cuda):
    """Instances that need no iteration, that stop early and that run long share a
    launch; each gives the bits of its own run."""
    import torch

    import shearwave_b200 as sw
    from shearwave_b200 import ops

    rng = np.random.default_rng(5)
    shapes = [(12, 11, 10), (3, 3, 3), (40, 33, 70), (9, 18, 34), (2, 5, 6), (33, 34, 66)]
    h, tols, iters = 0.5e-3, [1e-9, 1e-9, 1e-9, 1e-3, 1e-9, 1e-9], [500, 500, 500, 500, 500, 4]
    f = [[torch.as_tensor(rng.standard_normal(s), device=cuda) for _ in range(3)] for s in shapes]
    f[3] = [torch.zeros_like(c) for c in f[3]]  # divergence-free: early exit
    outs, stats = ops.project_batch([c[0] for c in f], [c[1] for c in f], [c[2] for c in f],
                                    [h] * 18, tols, iters)
    for k, s in enumerate(shapes):
        info = {}
        alone = sw.project_vector_field(*f[k], h, h, h, tols[k], iters[k], info=info)
        pz = ops.pitch(s[2])
        both = outs[k].reshape(3, s[0], s[1], pz)[..., :s[2]]
        assert all(torch.equal(a, b) for a, b in zip(alone, both)), k
        assert int(stats[k, 0]) == info["iters"]


@pytest.mark.parametrize("shape", [(69, 113, 147), (118, 105, 79)])
def test_repeats_are_bitwise(cuda, shape):
    # every sum is in a fixed order, so any difference is a race in the rings
    import torch

    import shearwave_b200 as sw

    g = torch.Generator(device="cuda").manual_seed(3)
    f = [torch.randn(shape, device=cuda, dtype=torch.float64, generator=g) for _ in range(3)]
    first = None
    for _ in range(60):
        out = sw.project_vector_field(*f, 5e-4, 5e-4, 5e-4, 1e-10, 300)
        first = [o.clone() for o in out] if first is None else first
        assert all(torch.equal(a, b) for a, b in zip(out, first))
