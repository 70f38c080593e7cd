"""Lone mixed solves in resident launches against plain launches, bit for bit.

Both run the same two-step tiles; resident launches only order them by their
neighbours' progress.  Grids with one tile, with chunks of two planes, with more
tiles than SMs, with both tile shapes; pushes, snapshots, damping; an odd last
step; runs of several launches.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(shape, n_steps, seed, graph, **more):
    import shearwave_b200 as sw

    rng = np.random.default_rng(seed)
    rho = (1000 * (1 + 0.05 * rng.uniform(-1, 1, shape))).astype(np.float32)
    mu = (3e3 * (1 + 0.3 * rng.uniform(-1, 1, shape))).astype(np.float32)
    opts = dict(env_t=(rng.uniform(size=n_steps) < 0.2).astype(np.float32), poisson_tol=1e-10,
                eta=more.pop("eta", 0.5), cuda_graph=graph,
                initial_u=rng.standard_normal((*shape, 3)).astype(np.float32), **more)
    stride = opts.pop("stride", None)
    b = rng.standard_normal(shape).astype(np.float32)
    h = 0.5e-3
    return sw.shear_fdtd(None, b, None, rho, mu, h, h, h, 1e-5, n_steps, opts,
                         snapshot_stride=stride)


@pytest.mark.parametrize("shape,n_steps,more", [
    ((3, 3, 3), 9, {}),
    ((9, 11, 20), 24, dict(stride=3)),
    ((64, 64, 64), 101, dict(stride=None)),
    ((40, 31, 61), 30, dict(vel_damp=0.01, stride=5)),
    ((21, 16, 130), 31, dict(eta=0.0)),
    ((6, 400, 320), 12, {}),            # more columns than SMs
    ((12, 300, 330), 21, dict(stride=7)),
    ((33, 29, 17), 1500, {}),           # several launches
])
def test_resident_matches_plain_launches(cuda, shape, n_steps, more):
    a = _solve(shape, n_steps, 7, True, **dict(more))
    b = _solve(shape, n_steps, 7, False, **dict(more))
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=True)


def test_compensation_planes_stay_zero(cuda):
    """The progress words live in a shell plane of the compensation component and
    leave it zero."""
    import torch

    from shearwave_b200 import solver as S

    b = torch.ones((20, 18, 24), device=cuda)
    sv = S._Solve(None, None, b, 1000.0, 2000.0, 1e-3, 1e-3, 1e-3, 1e-5, 40,
                  dict(env_t=np.ones(40, np.float32), poisson_tol=1e-10))
    S._project_inputs([sv])
    sv.build_terms()
    sv.run_loop(None)
    torch.cuda.synchronize()
    assert int(torch.count_nonzero(sv.run.state[:, 6:])) == 0
    assert sv.run.queue.tolist() == [0, 0]


def test_two_streams(cuda):
    """Two solves stepping at once on two streams keep their own progress."""
    import torch

    import shearwave_b200 as sw

    def run(seed):
        rng = np.random.default_rng(seed)
        b = torch.as_tensor(rng.standard_normal((48, 50, 60)).astype(np.float32), device=cuda)
        return sw.shear_fdtd(None, None, b, 1000.0, 2000.0, 1e-3, 1e-3, 1e-3, 1e-5, 300,
                             dict(env_t=np.ones(300, np.float32), poisson_tol=1e-10),
                             return_device=True)

    ref = [run(k) for k in (1, 2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = []
    for k, st in zip((1, 2), streams):
        with torch.cuda.stream(st):
            outs.append(run(k))
    torch.cuda.synchronize()
    for o, r in zip(outs, ref):
        assert all(torch.equal(x, y) for x, y in zip(o, r))


@pytest.mark.parametrize("shape,n_steps", [((64, 64, 64), 762), ((256, 256, 384), 48)])
def test_a_launch_holds_the_gpu_for_about_two_milliseconds(cuda, shape, n_steps):
    """Work on other streams waits for a resident launch, so its length is bounded."""
    import torch

    from shearwave_b200 import _native, ops
    from shearwave_b200 import solver as S

    b = torch.ones(shape, device=cuda)
    sv = S._Solve(None, None, b, 1000.0, 2000.0, 1e-3, 1e-3, 1e-3, 1e-5, n_steps,
                  dict(env_t=np.zeros(n_steps, np.float32), poisson_tol=1e-10))
    S._project_inputs([sv])
    sv.build_terms()
    sv.run_loop(None)  # warm
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    torch.cuda.synchronize()
    n = _native.launch_count()
    ends[0].record()
    ops.fdtd_steps_(*sv.run.bundle(), 0, n_steps)
    ends[1].record()
    torch.cuda.synchronize()
    assert ends[0].elapsed_time(ends[1]) / (_native.launch_count() - n) < 3.0


def test_a_pair_longer_than_the_bound(cuda):
    """Grids whose pairs take over 2 ms keep resident launches, of one pair each."""
    import torch

    from shearwave_b200 import _native
    from shearwave_b200 import solver as S

    n_steps, states = 6, []
    g = torch.Generator(device="cuda").manual_seed(3)
    b = torch.randn((512, 512, 500), device=cuda, generator=g)
    for resident in (True, False):
        sv = S._Solve(None, None, b, 1000.0, 2000.0, 1e-3, 1e-3, 1e-3, 1e-5, n_steps,
                      dict(env_t=np.ones(n_steps, np.float32), poisson_tol=1e-10))
        S._project_inputs([sv])
        sv.build_terms()
        if not resident:
            sv.run.queue = None
        n = _native.launch_count()
        sv.run_loop(None)
        torch.cuda.synchronize()
        assert n_steps // 2 <= _native.launch_count() - n < 10
        assert int(torch.count_nonzero(sv.run.state[:, 6:])) == 0
        states.append(sv.run.state)
    assert torch.equal(*states)
