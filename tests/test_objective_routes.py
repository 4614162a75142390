"""The route of the differentiable objective on the CPU: smoothing, warp and
filtering replaced by torch expressions, so that only the choice between the
fused pass and the torch form of the sum of squares is the package's."""
import numpy as np
import pytest
import torch
from torch.autograd import forward_ad

from broccoli_b200 import autograd as AG

SHAPE = (3, 4, 5)
FILTERS = [1.0, 2.0, -0.5]


class Fused(Exception):
    pass


@pytest.fixture
def stages(monkeypatch):
    def fused(*args):
        raise Fused

    monkeypatch.setattr(AG, "smooth3d", lambda v, sigma: v)
    monkeypatch.setattr(AG, "warp_affine", lambda v, p: v + p[0, 0])
    monkeypatch.setattr(AG, "filter3d", lambda v, f: torch.stack(
        [torch.stack([c * v, v + c], -1) for c in f], 1))
    monkeypatch.setattr(AG.FilterSsd, "apply", fused)


def _inputs(seed=0):
    gen = torch.Generator().manual_seed(seed)
    moving = torch.randn(SHAPE, generator=gen)
    q_ref = torch.randn((1, len(FILTERS)) + SHAPE + (2,), generator=gen)
    return moving, q_ref


def _objective(moving, q_ref):
    return AG.registration_objective(moving, q_ref, FILTERS, 1.0, params=torch.full((12,), 0.25))


def _plain(moving, q_ref):
    v = (moving + 0.25)[None]
    return ((torch.stack([torch.stack([c * v, v + c], -1) for c in FILTERS], 1) - q_ref) ** 2).sum()


def test_constant_reference_responses_take_the_fused_pass(stages):
    moving, q_ref = _inputs()
    with pytest.raises(Fused):
        _objective(moving, q_ref)
    with torch.no_grad(), pytest.raises(Fused):
        _objective(moving, q_ref.requires_grad_(True))


@pytest.mark.parametrize("f", [lambda x: x, torch.sqrt])
def test_second_derivatives_of_the_reference_responses(stages, f):
    moving, q_ref = _inputs()
    second = []
    for objective in (_objective, _plain):
        q = q_ref.clone().requires_grad_(True)
        g, = torch.autograd.grad(f(objective(moving, q)), q, create_graph=True)
        second.append((g.detach(),) + torch.autograd.grad((g ** 2).sum(), q))
    for a, b in zip(*second):
        assert torch.equal(a, b)


def test_forward_mode_tangents_of_the_reference_responses(stages):
    moving, q_ref = _inputs()
    t = torch.ones_like(q_ref)
    with forward_ad.dual_level():
        q = forward_ad.make_dual(q_ref, t)
        got, want = (forward_ad.unpack_dual(o(moving, q)).tangent for o in (_objective, _plain))
    assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16])
def test_fused_objective_refuses_host_tensors(dtype):
    """The fused operation hands raw pointers to the library: tensors that are
    not float32 on CUDA are refused before that, whatever the device."""
    bank = np.zeros((3, 2, 7, 7, 7), np.float32)
    vol = torch.zeros((1,) + SHAPE, dtype=dtype)
    with pytest.raises(TypeError):
        AG.FilterSsd.apply(vol, bank, torch.zeros((1, 3) + SHAPE + (2,), dtype=dtype))


class Halved(torch.Tensor):
    """Responses stored at twice their value: subtraction reads the half."""

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        plain = [a.as_subclass(torch.Tensor) if isinstance(a, Halved) else a for a in args]
        if func in (torch.Tensor.sub, torch.Tensor.__sub__, torch.sub):
            plain[1] = 0.5 * plain[1]
        return func(*plain, **(kwargs or {}))


def test_reference_responses_with_operations_of_their_own(stages):
    """Tensor subclasses and sparse tensors take the torch form, which calls
    their operations."""
    moving, q_ref = _inputs()
    want = _plain(moving, q_ref)
    assert torch.equal(_objective(moving, (2.0 * q_ref).as_subclass(Halved)), want)
    assert torch.equal(_objective(moving, q_ref.to_sparse()), want)
