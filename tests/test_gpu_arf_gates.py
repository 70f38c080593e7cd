"""Radiation force over record lengths, gates, alignments and types.

Sums run in float64 on both sides.  With n gated samples they differ by at
most about n eps of the sum of |p v|, so float64 results agree to 1e-13 of
the mean |p v| scale (n < 400) and float32 ones to the rounding of the output.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(p, q, c, rho, alpha, f0, idx):
    pv = p[..., idx].astype(np.float64) * q[..., idx].astype(np.float64)
    alpha_np = alpha * (f0 / 1e6) / 8.685889638 * 100.0
    scale = np.abs(pv).mean(-1)
    if p is q:
        return 2 * alpha_np * (pv.mean(-1) / (rho * c)) / c, 2 * alpha_np * scale / (rho * c) / c
    return 2 * alpha_np / c * pv.mean(-1), 2 * alpha_np / c * scale


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nt", [1, 3, 17, 32, 257, 300, 1030])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 5, 7), (9, 8, 33)])
def test_gates(cuda, shape, nt, dtype):
    import torch

    import shearwave_b200 as sw

    rng = np.random.default_rng(nt + sum(shape))
    n = int(np.prod(shape)) * nt
    # bases on a 16-byte boundary and one element past it
    whole = [torch.as_tensor(rng.standard_normal(n + 1).astype(dtype), device=cuda)
             for _ in range(4)]
    gates = [slice(0, nt), slice(nt // 3, nt // 3 + max(1, nt // 2)),
             np.arange(0, nt, 3), np.r_[nt - 1, 0], np.arange(nt)[::-1]]
    tol = 1e-13 if dtype == np.float64 else 1.2e-7
    for off in (0, 1):
        rec = [w[off: off + n].reshape(*shape, nt) for w in whole]
        host = [r.cpu().numpy() for r in rec]
        for gate in gates:
            idx = np.arange(nt)[gate] if isinstance(gate, slice) else gate
            out = sw.compute_radiation_force(rec[0], 1540.0, 1000.0, 0.5, 5e6, gate=gate)
            ref, scale = _reference(host[0], host[0], 1540.0, 1000.0, 0.5, 5e6, idx)
            assert np.all(np.abs(out.cpu().numpy() - ref) <= tol * scale)
            outs = sw.compute_radiation_force_velocity(*rec, 1540.0, 1000.0, 0.5, 5e6, gate=gate)
            for o, v in zip(outs, host[1:]):
                ref, scale = _reference(host[0], v, 1540.0, 1000.0, 0.5, 5e6, idx)
                assert np.all(np.abs(o.cpu().numpy() - ref) <= tol * scale)
    # records whose alignments differ
    mix = [whole[0][:n].reshape(*shape, nt)] + [w[1:].reshape(*shape, nt) for w in whole[1:]]
    outs = sw.compute_radiation_force_velocity(*mix, 1540.0, 1000.0, 0.5, 5e6, gate=slice(0, nt))
    for o, v in zip(outs, mix[1:]):
        ref, scale = _reference(mix[0].cpu().numpy(), v.cpu().numpy(), 1540.0, 1000.0, 0.5, 5e6,
                                np.arange(nt))
        assert np.all(np.abs(o.cpu().numpy() - ref) <= tol * scale)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nt", [1, 31, 300, 341, 342, 513, 1024, 1025, 2100])
@pytest.mark.parametrize("ncell", [1, 37, 5000])
def test_envelope(cuda, ncell, nt, dtype):
    import torch

    from shearwave_b200 import ops

    rng = np.random.default_rng(nt + ncell)
    p = rng.standard_normal((ncell, nt)).astype(dtype)
    env = ops.arf_envelope(torch.as_tensor(p, device=cuda), ncell, nt).cpu().numpy()
    ref = (p.astype(np.float64) ** 2).mean(0)
    assert np.all(np.abs(env - ref) <= 1e-12 * ref)


@pytest.mark.parametrize("gate", [slice(2, 30), slice(5, 85), slice(0, 100), slice(0, 109)])
def test_several_rounds_per_warp(cuda, gate):
    # enough cells that a warp takes more than one round of every lane split,
    # the last one partly empty; at most 109 samples: the same bound
    import torch

    import shearwave_b200 as sw

    shape, nt = (33, 41, 37), 109
    rng = np.random.default_rng(gate.stop)
    host = [rng.standard_normal((*shape, nt)) for _ in range(4)]
    rec = [torch.as_tensor(h, device=cuda) for h in host]
    idx = np.arange(nt)[gate]
    out = sw.compute_radiation_force(rec[0], 1540.0, 1000.0, 0.5, 5e6, gate=gate)
    ref, scale = _reference(host[0], host[0], 1540.0, 1000.0, 0.5, 5e6, idx)
    assert np.all(np.abs(out.cpu().numpy() - ref) <= 1e-13 * scale)
    outs = sw.compute_radiation_force_velocity(*rec, 1540.0, 1000.0, 0.5, 5e6, gate=gate)
    for o, v in zip(outs, host[1:]):
        ref, scale = _reference(host[0], v, 1540.0, 1000.0, 0.5, 5e6, idx)
        assert np.all(np.abs(o.cpu().numpy() - ref) <= 1e-13 * scale)
