"""The strain post-pass and the operators bit for bit at tile edges, in strided
inputs, on unaligned tensors, and over the whole exponent range (the division
by the spacing is a multiply-add sequence inside a range of exponents and a
division outside it)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (1, 4, 5), (13, 8, 32), (12, 9, 33), (25, 17, 65), (5, 1, 40), (14, 10, 2)]
H = (0.5e-3, 0.37e-3, 0.71e-3)


def _field(rng, shape, dtype, wide):
    f = rng.standard_normal(shape)
    if wide:  # from subnormal to overflowing quotients, with exact and signed zeros
        top = 40 if dtype == np.float32 else 310
        f = f * 10.0 ** rng.uniform(-top - 8, top - 4, shape)
        f[rng.uniform(size=shape) < 0.2] = 0.0
        f[rng.uniform(size=shape) < 0.1] = -0.0
    with np.errstate(all="ignore"):
        return f.astype(dtype)


def _same(a, b):
    np.testing.assert_array_equal(a, b)
    zero = (b == 0) & np.isfinite(b)
    assert np.array_equal(np.signbit(a[zero]), np.signbit(b[zero]))


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_strain_and_operators_bitwise(cuda, shape, dtype, wide):
    import shearwave_b200 as sw
    from oracle import shearwave_oracle as O

    rng = np.random.default_rng(sum(shape) + wide)
    u = [_field(rng, shape, dtype, wide) for _ in range(3)]
    with np.errstate(all="ignore"):
        eps = O.compute_strain_tensor(*u, *H)
        inv = O.compute_strain_invariants(eps)
        # the kernels clamp a NaN second invariant to 0 (numpy's maximum keeps it)
        inv["max_shear"] = np.where(np.isnan(inv["max_shear"]), dtype(0), inv["max_shear"])
        lap, div = O.laplacian_center(u[0], *H), O.divergence_center(*u, *H)
        grad = O.gradient_center(u[0], *H)
    _same(sw.compute_strain_tensor(*u, *H), eps)
    e2, i2 = sw.compute_strain_fields(np.stack(u, -1), *H)
    _same(e2, eps)
    for k, v in inv.items():
        _same(i2[k], v)
        _same(sw.compute_strain_invariants(eps)[k], v)
    _same(sw.laplacian_center(u[0], *H), lap)
    _same(sw.divergence_center(*u, *H), div)
    for a, b in zip(sw.gradient_center(u[0], *H), grad):
        _same(a, b)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_invariants_of_an_unaligned_tensor(cuda, dtype):
    import torch

    import shearwave_b200 as sw
    from oracle import shearwave_oracle as O

    rng = np.random.default_rng(3)
    flat = torch.as_tensor(rng.standard_normal(6 * 333 + 1).astype(dtype), device=cuda)
    eps = flat[1:].reshape(333, 6)
    ref = O.compute_strain_invariants(eps.cpu().numpy())
    for k, v in sw.compute_strain_invariants(eps).items():
        _same(v.cpu().numpy(), ref[k])
