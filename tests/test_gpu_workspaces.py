"""The C entries that take a workspace, at every alignment of it."""

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

SHAPE, H = (11, 14, 21), 0.5e-3


@pytest.fixture(scope="module")
def fields(cuda):
    import torch

    g = torch.Generator(device="cuda").manual_seed(2)
    return [torch.randn(SHAPE, device=cuda, dtype=torch.float64, generator=g) for _ in range(3)]


@pytest.mark.parametrize("offset", [0, 4, 8, 16, 48, 64, 72, 120, 128])
@pytest.mark.parametrize("entry", ["sw_project", "sw_project_spectral", "sw_static_solve"])
def test_workspace_at_any_address(cuda, fields, entry, offset):
    import torch

    from shearwave_b200 import _native, ops

    nx, ny, nz = SHAPE
    lib = _native.load()
    query = lib.sw_project_spectral_workspace_bytes if "spectral" in entry else \
        lib.sw_project_workspace_bytes
    nb = int(query(nx, ny, nz))
    # bytes on both sides of the workspace that no kernel may touch
    room = torch.full((nb + 512,), 0x5A, dtype=torch.uint8, device=cuda)
    at = 256 + offset
    ncomp = 1 if entry == "sw_static_solve" else 3
    out = torch.empty((ncomp, nx, ny, ops.pitch(nz)), dtype=torch.float64, device=cuda)
    st = _native.CGStats()
    f = [c.data_ptr() for c in fields]
    grid = (ny * nz, nz, 1, nx, ny, nz, H, H, H)
    tail = (out.data_ptr(), room.data_ptr() + at, nb, C.byref(st),
            torch.cuda.current_stream().cuda_stream)
    if entry == "sw_project":
        _native.call(entry, _native.SW_F64, *f, *grid, 1e-9, 200, *tail)
        ref, _ = ops.project(*fields, [H] * 3, 1e-9, 200, "cg")
    elif entry == "sw_project_spectral":
        _native.call(entry, _native.SW_F64, *f, *grid, *tail)
        ref, _ = ops.project(*fields, [H] * 3, 1e-9, 200, "spectral")
    else:
        _native.call(entry, _native.SW_F64, f[0], None, 2.0, *grid, 1e-9, 200, *tail)
        ref, _ = ops.static_solve(fields[0], None, 2.0, [H] * 3, 1e-9, 200)
    assert torch.equal(out.reshape(ncomp, -1)[:, :nx * ny * ops.pitch(nz)],
                       ref.reshape(ncomp, -1))
    assert bool((room[:at] == 0x5A).all()) and bool((room[at + nb:] == 0x5A).all())
