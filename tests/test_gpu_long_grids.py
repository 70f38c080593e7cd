"""Grids longer than a launch's 65535 blocks along y or x, and records longer than that
many chunks of samples."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(262145, 1, 3), (1, 524281, 2), (262141, 2, 33)])
def test_convert(cuda, shape):
    import torch

    from shearwave_b200 import ops

    nx, ny, nz = shape
    g = torch.Generator(device="cuda").manual_seed(4)
    src = torch.randn((nx, ny, ops.pitch(nz)), device=cuda, dtype=torch.float64, generator=g)
    dst = torch.full(shape, -7.0, device=cuda)
    ops.convert_(dst, src.reshape(-1), 1, list(shape), [0, ny * nz, nz, 1], 0.5, None, [0, 0, 0])
    assert torch.equal(dst, (src[..., :nz] * 0.5).float())


def test_convert_in_strides_with_densities(cuda):
    # two components into a (nx, ny, nz, 2) array, divided by a map's density
    import torch

    from shearwave_b200 import ops

    nx, ny, nz = 262142, 3, 2
    g = torch.Generator(device="cuda").manual_seed(9)
    src = torch.randn((2, nx, ny, ops.pitch(nz)), device=cuda, dtype=torch.float64, generator=g)
    rho = torch.rand((nx, ny, nz), device=cuda, dtype=torch.float64, generator=g) + 0.5
    dst = torch.empty((nx, ny, nz, 2), device=cuda, dtype=torch.float64)
    ops.convert_(dst, src.reshape(-1), 2, [nx, ny, nz], [1, ny * nz * 2, nz * 2, 2], 1.0, rho,
                 [ny * nz, nz, 1])
    assert torch.equal(dst, (src[..., :nz] * (1.0 / rho)).permute(1, 2, 3, 0).contiguous())


@pytest.mark.parametrize("shape", [(786421, 3, 3), (65536, 4, 3)])
def test_strain(cuda, shape):
    import shearwave_b200 as sw
    from oracle import shearwave_oracle as O

    rng = np.random.default_rng(6)
    u = rng.standard_normal((*shape, 3), dtype=np.float32)
    h = (0.5e-3, 0.37e-3, 0.71e-3)
    ref = O.compute_strain_tensor(*np.moveaxis(u, -1, 0), *h)
    eps, inv = sw.compute_strain_fields(u, *h)
    assert np.array_equal(eps, ref)
    for k, v in O.compute_strain_invariants(ref).items():
        assert np.array_equal(inv[k], v), k


@pytest.mark.parametrize("ncell", [1, 3])
def test_envelope(cuda, ncell):
    import torch

    from shearwave_b200 import ops

    nt = 65535 * 1024 + 5
    g = torch.Generator(device="cuda").manual_seed(8)
    p = torch.randint(-8, 9, (ncell, nt), device=cuda, generator=g, dtype=torch.int8).float()
    env = ops.arf_envelope(p, ncell, nt)
    # whole numbers: every sum is exact, the division rounded once (by numpy: torch
    # multiplies by the reciprocal)
    assert np.array_equal(env.cpu().numpy(), (p.double() ** 2).sum(0).cpu().numpy() / ncell)
