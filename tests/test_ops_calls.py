"""The package's calls of its operators (no GPU): modes still see them, gradients
and written arguments are treated as by the operators themselves."""

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.utils._python_dispatch import TorchDispatchMode

from shearwave_b200 import ops


class _Log(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(func)
        return func(*args, **(kwargs or {}))


def test_a_mode_sees_the_call_and_fakes_have_shapes():
    with FakeTensorMode():
        f = torch.empty((5, 6, 7), device="cuda")
        with _Log() as log:
            out = ops.laplacian(f, [1.0, 1.0, 1.0])
    assert torch.ops.shearwave_b200.laplacian.default in log.seen
    assert out.shape == f.shape


def test_cpu_tensors_are_refused():
    with pytest.raises(NotImplementedError):
        ops.laplacian(torch.zeros(4, 4, 4), [1.0, 1.0, 1.0])


@pytest.mark.parametrize("call", [ops.laplacian, torch.ops.shearwave_b200.laplacian.default])
def test_no_gradient_formula(call):
    with FakeTensorMode():
        f = torch.empty((5, 6, 7), device="cuda", requires_grad=True)
        out = call(f, [1.0, 1.0, 1.0])
        assert out.requires_grad
        with pytest.raises(RuntimeError):
            out.sum().backward()
        with torch.no_grad():
            assert not call(f, [1.0, 1.0, 1.0]).requires_grad


@pytest.mark.parametrize("call", [ops.convert_, torch.ops.shearwave_b200.convert_.default])
def test_written_arguments_get_a_new_version(call):
    with FakeTensorMode():
        dst = torch.empty((4, 4, 4), device="cuda")
        src = torch.empty((128,), device="cuda", dtype=torch.float64)
        v0, s0 = dst._version, src._version
        call(dst, src, 1, [4, 4, 4], [0, 16, 4, 1], 1.0, None, [0, 0, 0])
        assert dst._version == v0 + 1 and src._version == s0


def test_keyword_arguments():
    with FakeTensorMode():
        f = torch.empty((5, 6, 7), device="cuda")
        assert ops.laplacian(f=f, h=[1.0, 1.0, 1.0]).shape == f.shape
        assert ops.laplacian(f, h=[1.0, 1.0, 1.0]).shape == f.shape
        out, st = ops.project(fx=f, fy=None, fz=None, h=[1.0] * 3, tol=1e-8, max_iters=4,
                              method="cg")
        assert out.shape == (3, 5 * 6 * 8) and st.shape == (4,)
        dst = torch.empty((4, 4, 4), device="cuda")
        v = dst._version
        ops.convert_(dst=dst, src=torch.empty(128, device="cuda", dtype=torch.float64), ncomp=1,
                     shape=[4, 4, 4], dst_strides=[0, 16, 4, 1], scale=1.0, rho=None,
                     rho_strides=[0, 0, 0])
        assert dst._version == v + 1
    with pytest.raises(RuntimeError):
        ops.laplacian(f, g=f)
