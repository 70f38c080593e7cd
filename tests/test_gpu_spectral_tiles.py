"""The direct projection at chain lengths around its tiles of 32 modes.

The oracle builds each axis's operator as a matrix and solves with its
eigendecomposition (numpy, float64).  Each transform sums at most K products,
so six of them and the division leave an error of about
6 K eps sqrt(lmax / lmin) of the force's norm: below 1e-10 for n <= 300.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _project(f, h):
    shape = f[0].shape
    inner = (slice(1, -1),) * 3
    m = np.zeros(shape)
    m[inner] = 1.0
    f = [c * m for c in f]
    grads, lams, qs = [], [], []
    for n, d in zip(shape, h):
        g = np.zeros((n, n))
        i = np.arange(1, n - 1)
        g[i, i + 1], g[i, i - 1] = 1 / (2 * d), -1 / (2 * d)
        lam, q = np.linalg.eigh(-(g @ g)[1:-1, 1:-1])
        grads.append(g)
        lams.append(lam)
        qs.append(q)

    def diff(a, axis):
        return np.moveaxis(np.tensordot(grads[axis], a, (1, axis)), 0, axis) * m

    b = -sum(diff(c, a) for a, c in enumerate(f))[inner]
    for q in qs:
        b = np.tensordot(b, q, ([0], [0]))
    total = lams[0][:, None, None] + lams[1][None, :, None] + lams[2][None, None, :]
    ok = total > 1e-12 * total.max()
    b = np.where(ok, b / np.where(ok, total, 1.0), 0.0)
    for q in qs:
        b = np.tensordot(b, q.T, ([0], [0]))
    phi = np.zeros(shape)
    phi[inner] = b
    return [c - diff(phi, a) for a, c in enumerate(f)]


# chains of 1, 16, 31-33, 64/65, 96/97, 128/129 and 149 modes on each axis, both parities
@pytest.mark.parametrize("shape", [
    (3, 4, 5), (4, 3, 34), (64, 66, 65), (68, 7, 131), (6, 132, 67), (195, 9, 8), (10, 196, 33),
    (7, 6, 194), (258, 5, 6), (5, 260, 7), (6, 5, 259), (9, 8, 300),
])
def test_direct_projection_at_tile_edges(cuda, shape):
    import shearwave_b200 as sw

    rng = np.random.default_rng(sum(shape))
    h = (0.5e-3, 0.4e-3, 0.7e-3)
    f = [rng.standard_normal(shape) for _ in range(3)]
    out = sw.project_vector_field(*f, *h, 0.0, 0, method="spectral")
    ref = _project(f, h)
    norm = np.sqrt(sum(np.sum(c * c) for c in f))
    err = np.sqrt(sum(np.sum((a - b) ** 2) for a, b in zip(out, ref)))
    assert err <= 1e-10 * norm, err / norm
