"""Differentiable registration: gradients of the filter-response SSD with
respect to the 12 affine parameters and to a displacement field, from the
adjoint kernels through torch.autograd, against central finite differences
of the FP64 oracle with a step of 1e-3 voxel (translations and field
values 1e-3; an affine matrix entry the step that moves no voxel by more
than 1e-3 voxel).  Bar: relative error <= 1e-3,
|g_gpu - g_fd| <= 1e-3 * max|g_fd| over the checked components.

Evaluated away from the grid (sub-voxel parameters / field) so that the
trilinear interpolant is differentiable at every sample point."""
import numpy as np
import pytest
import torch

from broccoli_b200 import autograd as AG
from broccoli_b200 import synthetic as S

pytestmark = pytest.mark.gpu
H_FD = 1e-3
SIGMA = 2.0
SHAPE = (20, 26, 24)


def _pair():
    sub, tpl, _ = S.t1_template_pair(SHAPE, SHAPE, seed=3)
    return sub.astype(np.float32), tpl.astype(np.float32)


def _fd_steps(shape):
    """Central-difference steps of the 12 parameters that move no voxel by
    more than 1e-3 voxel: 1e-3 for the translations, 1e-3 / (half extent of
    the coordinate it multiplies) for a matrix entry (column 0 multiplies
    x - (W-1)/2, column 1 y, column 2 z)."""
    D, H, W = shape
    half = [(W - 1) / 2.0, (H - 1) / 2.0, (D - 1) / 2.0]
    return np.array([H_FD] * 3 + [H_FD / half[(i - 3) % 3] for i in range(3, 12)])


def _params():
    p = np.zeros(12, np.float64)
    p[:3] = [0.31, -0.27, 0.43]
    p[3:] = np.array([0.011, -0.007, 0.004, 0.006, -0.013, 0.002, -0.005, 0.008, 0.009])
    return p


def test_filter_adjoint_is_the_transpose(ctx, lin_filters):
    """<F x, y> == <x, F^T y> for random x, y."""
    rng = np.random.default_rng(0)
    x = torch.from_numpy(rng.standard_normal((2,) + SHAPE).astype(np.float32)).cuda()
    y = torch.from_numpy(rng.standard_normal((2, 3) + SHAPE + (2,)).astype(np.float32)).cuda()
    xr = x.clone().requires_grad_(True)
    fx = AG.filter3d(xr, lin_filters)
    lhs = (fx.double() * y.double()).sum()
    lhs.backward()
    rhs = (x.double() * xr.grad.double()).sum()
    assert abs(float(lhs) - float(rhs)) <= 1e-4 * abs(float(lhs))


def test_affine_gradient_vs_fp64_finite_differences(orc, lin_filters):
    mov, ref = _pair()
    dev = torch.device("cuda")
    q_ref = AG.reference_responses(torch.from_numpy(ref).to(dev), lin_filters, SIGMA)
    p = torch.tensor(_params(), dtype=torch.float32, device=dev, requires_grad=True)
    loss = AG.registration_objective(torch.from_numpy(mov).to(dev), q_ref, lin_filters, SIGMA, params=p)
    loss.backward()
    g = p.grad.cpu().numpy().astype(np.float64)
    p0 = _params()
    steps = _fd_steps(mov.shape)
    fd = np.zeros(12)
    for i in range(12):
        e = np.zeros(12)
        e[i] = steps[i]
        fd[i] = (orc.registration_objective(mov, ref, lin_filters, SIGMA, params=p0 + e) -
                 orc.registration_objective(mov, ref, lin_filters, SIGMA, params=p0 - e)) / (2 * steps[i])
    assert np.abs(g - fd).max() <= 1e-3 * np.abs(fd).max(), (g, fd)


def test_field_gradient_vs_fp64_finite_differences(orc, lin_filters):
    mov, ref = _pair()
    dev = torch.device("cuda")
    rng = np.random.default_rng(1)
    field = (rng.uniform(-0.45, 0.45, (3,) + SHAPE) + 0.05).astype(np.float64)
    q_ref = AG.reference_responses(torch.from_numpy(ref).to(dev), lin_filters, SIGMA)
    f = torch.tensor(field, dtype=torch.float32, device=dev, requires_grad=True)
    loss = AG.registration_objective(torch.from_numpy(mov).to(dev), q_ref, lin_filters, SIGMA, field=f)
    loss.backward()
    g = f.grad.cpu().numpy().astype(np.float64)
    # a seeded random subset of interior voxels, all three components
    D, H, W = SHAPE
    picks = [(c, rng.integers(4, D - 4), rng.integers(4, H - 4), rng.integers(4, W - 4))
             for c in range(3) for _ in range(3)]
    fd, gg = [], []
    for c, z, y, x in picks:
        fp = field.copy()
        fm = field.copy()
        fp[c, z, y, x] += H_FD
        fm[c, z, y, x] -= H_FD
        fd.append((orc.registration_objective(mov, ref, lin_filters, SIGMA, field=fp) -
                   orc.registration_objective(mov, ref, lin_filters, SIGMA, field=fm)) / (2 * H_FD))
        gg.append(g[c, z, y, x])
    fd = np.array(fd)
    gg = np.array(gg)
    assert np.abs(gg - fd).max() <= 1e-3 * np.abs(fd).max(), (gg, fd)


def test_moving_volume_gradient_vs_finite_differences(orc, lin_filters):
    """Gradient with respect to the moving volume (smoothing adjoint +
    scatter adjoint of the warp), checked at a few voxels."""
    mov, ref = _pair()
    dev = torch.device("cuda")
    q_ref = AG.reference_responses(torch.from_numpy(ref).to(dev), lin_filters, SIGMA)
    m = torch.from_numpy(mov).to(dev).requires_grad_(True)
    p = torch.tensor(_params(), dtype=torch.float32, device=dev)
    loss = AG.registration_objective(m, q_ref, lin_filters, SIGMA, params=p)
    loss.backward()
    g = m.grad.cpu().numpy().astype(np.float64)
    mv = mov.astype(np.float64)
    fd, gg = [], []
    h = 1e-2
    for z, y, x in [(10, 13, 12), (8, 9, 15), (12, 17, 7)]:
        a = mv.copy()
        b = mv.copy()
        a[z, y, x] += h
        b[z, y, x] -= h
        fd.append((orc.registration_objective(a, ref, lin_filters, SIGMA, params=_params()) -
                   orc.registration_objective(b, ref, lin_filters, SIGMA, params=_params())) / (2 * h))
        gg.append(g[z, y, x])
    fd = np.array(fd)
    assert np.abs(np.array(gg) - fd).max() <= 1e-3 * np.abs(fd).max()


def test_gradients_at_full_config_size(orc, lin_filters):
    """The differentiable-registration workload's own size: a 128x128x96 pair
    made as the T1-like template pair, smoothing sigma 2.  All 12 affine
    gradients and the field gradient at six seeded interior voxels (all
    three components) against FP64 central differences of the oracle (steps
    of 1e-3 voxel); bar 1e-3 of the largest finite difference, as above."""
    shape = (96, 128, 128)
    sub, tpl, _ = S.t1_template_pair(shape, shape, seed=3)
    mov, ref = sub.astype(np.float32), tpl.astype(np.float32)
    dev = torch.device("cuda")
    q_ref = AG.reference_responses(torch.from_numpy(ref).to(dev), lin_filters, SIGMA)
    p = torch.tensor(_params(), dtype=torch.float32, device=dev, requires_grad=True)
    AG.registration_objective(torch.from_numpy(mov).to(dev), q_ref, lin_filters, SIGMA, params=p).backward()
    g = p.grad.cpu().numpy().astype(np.float64)
    p0 = _params()
    steps = _fd_steps(mov.shape)
    fd = np.zeros(12)
    for i in range(12):
        e = np.zeros(12)
        e[i] = steps[i]
        fd[i] = (orc.registration_objective(mov, ref, lin_filters, SIGMA, params=p0 + e) -
                 orc.registration_objective(mov, ref, lin_filters, SIGMA, params=p0 - e)) / (2 * steps[i])
    assert np.abs(g - fd).max() <= 1e-3 * np.abs(fd).max(), (g, fd)

    rng = np.random.default_rng(7)
    field = (rng.uniform(-0.45, 0.45, (3,) + shape) + 0.05).astype(np.float64)
    f = torch.tensor(field, dtype=torch.float32, device=dev, requires_grad=True)
    AG.registration_objective(torch.from_numpy(mov).to(dev), q_ref, lin_filters, SIGMA, field=f).backward()
    gf = f.grad.cpu().numpy().astype(np.float64)
    D, H, W = shape
    picks = [(c, int(rng.integers(8, D - 8)), int(rng.integers(8, H - 8)), int(rng.integers(8, W - 8)))
             for c in range(3) for _ in range(2)]
    fdf, gg = [], []
    for c, z, y, x in picks:
        fp, fm = field.copy(), field.copy()
        fp[c, z, y, x] += H_FD
        fm[c, z, y, x] -= H_FD
        fdf.append((orc.registration_objective(mov, ref, lin_filters, SIGMA, field=fp) -
                    orc.registration_objective(mov, ref, lin_filters, SIGMA, field=fm)) / (2 * H_FD))
        gg.append(gf[c, z, y, x])
    fdf, gg = np.array(fdf), np.array(gg)
    assert np.abs(gg - fdf).max() <= 1e-3 * np.abs(fdf).max(), (gg, fdf)


@pytest.mark.parametrize("shape", [(1, 1, 1), (4, 16, 32), (5, 17, 33), (3, 31, 65), (9, 15, 31)])
@pytest.mark.parametrize("nf", [3, 6])
@pytest.mark.parametrize("offset", [0, 1])
def test_filter_adjoint_tile_edges(shape, nf, offset, bank):
    """brc_filter3d_adjoint at the edges of its 32 x 16 x 4 blocks, two
    volumes, with a gradient that is 8-byte aligned and one that is not,
    against the transpose of the convolution in FP64 (torch on the CPU): the
    adjoint is the cross-correlation with the unflipped filters.  FP32 bar of
    the suite, 1e-4 of the largest value."""
    flt = bank["linear" if nf == 3 else "nonlinear"]
    D, H, W = shape
    gen = torch.Generator().manual_seed(sum(shape) + nf)
    g = torch.randn((2, nf) + shape + (2,), generator=gen)
    ref = torch.nn.functional.conv3d(
        torch.movedim(g.double(), -1, 2).reshape(2, 2 * nf, D, H, W),
        torch.from_numpy(flt).double().reshape(1, 2 * nf, 7, 7, 7), padding=3)[:, 0]
    buf = torch.empty(g.numel() + 1, device="cuda")
    gd = buf[offset:offset + g.numel()]
    gd.copy_(g.reshape(-1))
    out = torch.full((2,) + shape, float("nan"), device="cuda")
    c = AG._ctx(out.device)
    fn = AG._sig("brc_filter3d_adjoint", [AG._P, AG._P, AG._I, AG._I, AG._I, AG._I, AG._P, AG._I, AG._P])
    f = np.ascontiguousarray(flt, np.float32)
    assert fn(c.handle, AG._p(gd), W, H, D, 2, f.ctypes.data, nf, AG._p(out)) == 0
    err = (out.cpu().double() - ref).abs().max() / ref.abs().max()
    assert float(err) < 1e-4


@pytest.mark.parametrize("shape", [(3, 5, 7), (6, 9, 8), (12, 16, 20)])
@pytest.mark.parametrize("offset", [0, 1])
def test_objective_equals_its_torch_form(shape, offset, lin_filters):
    """The fused residual and sum of squares against the same objective from
    the filtering and torch's elementwise operations: loss, gradient of the
    parameters and of the reference responses (FilterSsd itself; the objective
    takes the torch form for these), with reference responses that are 16-byte
    aligned and that are not.  Both sum FP32 squares of the same residuals in
    another order: 1e-5 relative.  A second backward pass raises."""
    gen = torch.Generator().manual_seed(sum(shape))
    moving = (torch.randn(shape, generator=gen) * 50 + 100).cuda()
    q = AG.reference_responses((torch.randn(shape, generator=gen) * 50 + 100).cuda(), lin_filters, SIGMA)
    buf = torch.empty(q.numel() + offset, device="cuda")
    buf[offset:].copy_(q.reshape(-1))
    grads = []
    for fused in (True, False):
        p = torch.tensor(_params(), dtype=torch.float32, device="cuda", requires_grad=True)
        q_ref = buf[offset:].reshape(q.shape).detach()
        if fused:
            objective = AG.registration_objective(moving, q_ref, lin_filters, SIGMA, params=p).detach()
        q_ref.requires_grad_(True)
        w = AG.warp_affine(AG.smooth3d(moving[None], SIGMA), p.reshape(1, 12))
        loss = AG.FilterSsd.apply(w, lin_filters, q_ref) if fused else ((AG.filter3d(w, lin_filters) - q_ref) ** 2).sum()
        if fused:
            assert torch.equal(loss.detach(), objective)
            g, = torch.autograd.grad(torch.sqrt(loss), q_ref, create_graph=True)
            with pytest.raises(RuntimeError, match="once_differentiable"):
                g.sum().backward()
            loss = AG.FilterSsd.apply(w, lin_filters, q_ref)
        grads.append((loss.detach(),) + torch.autograd.grad(3.0 * loss, (p, q_ref)))
    for a, b in zip(*grads):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


def _objective_inputs(shape, seed, lin_filters):
    gen = torch.Generator().manual_seed(seed)
    moving = (torch.randn(shape, generator=gen) * 50 + 100).cuda()
    q = AG.reference_responses((torch.randn(shape, generator=gen) * 50 + 100).cuda(), lin_filters, SIGMA)
    field = (torch.rand((3,) + tuple(shape), generator=gen) - 0.5).cuda()
    return moving, q, field


def test_objective_keeps_no_sums_in_the_shared_context(lin_filters, monkeypatch):
    """One context serves every stream of a device, so the objective may hold
    no per-call sums in it: a field objective, and the affine gradient, after a
    filtering and a smoothing of the same volume leave the context's workspace
    as it was."""
    monkeypatch.setattr(AG, "_contexts", {})
    moving, q, field = _objective_inputs((9, 12, 10), 5, lin_filters)
    before = AG._ctx(moving.device).workspace_bytes
    AG.registration_objective(moving, q, lin_filters, SIGMA, field=field)
    assert AG._ctx(moving.device).workspace_bytes == before
    p = torch.tensor(_params(), dtype=torch.float32, device="cuda", requires_grad=True)
    AG.warp_affine(moving[None], p.reshape(1, 12)).sum().backward()
    assert AG._ctx(moving.device).workspace_bytes == before


@pytest.mark.parametrize("form", ["field", "params"])
def test_objectives_on_two_streams(form, lin_filters):
    """Objectives and their gradients queued alternately on two streams, the
    large and the small one of each round free to run at once, give the results
    of calls that run alone, bit for bit (a fixed order of sums)."""
    cases = [_objective_inputs(s, i, lin_filters) for i, s in enumerate([(40, 64, 64), (12, 20, 16)])]

    def step(m, q, f):
        x = (f if form == "field" else torch.tensor(_params(), dtype=torch.float32, device="cuda")).requires_grad_(True)
        loss = AG.registration_objective(m, q, lin_filters, SIGMA, **{form: x})
        return torch.cat([loss.detach().reshape(1), torch.autograd.grad(loss, x)[0].reshape(-1)])

    alone = []
    for c in cases:
        alone.append(step(*c))
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    outs = []
    for _ in range(20):
        for (m, q, f), s in zip(cases, streams):
            with torch.cuda.stream(s):
                outs.append(step(m, q, f))
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        assert torch.equal(out, alone[k % 2])


@pytest.mark.parametrize("form", ["field", "params"])
def test_captured_objective_outlives_later_calls(form, lin_filters, monkeypatch):
    """An objective and its gradient captured in a CUDA graph replay to the
    eager results after calls that make the context grow: they hold no memory
    of the context."""
    monkeypatch.setattr(AG, "_contexts", {})
    m, q, f = _objective_inputs((10, 14, 12), 3, lin_filters)
    x = (f if form == "field" else torch.tensor(_params(), dtype=torch.float32, device="cuda")).requires_grad_(True)

    def step():
        loss = AG.registration_objective(m, q, lin_filters, SIGMA, **{form: x})
        return (loss.detach(),) + torch.autograd.grad(loss, x)

    eager = step()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        step()
    torch.cuda.current_stream().wait_stream(stream)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = step()
    m2, q2, _ = _objective_inputs((40, 64, 64), 4, lin_filters)
    p = torch.tensor(_params(), dtype=torch.float32, device="cuda", requires_grad=True)
    AG.registration_objective(m2, q2, lin_filters, SIGMA, params=p).backward()
    AG._ctx(m.device).register_linear(m2, m2[None].repeat(8, 1, 1, 1), lin_filters, 1)  # larger partial rows
    g.replay()
    torch.cuda.synchronize()
    for a, b in zip(captured, eager):
        assert torch.equal(a, b)


@pytest.mark.parametrize("vol, ref, error", [
    (torch.float64, torch.float32, TypeError), (torch.float16, torch.float32, TypeError),
    (torch.float32, torch.float64, TypeError), (torch.float32, torch.float16, TypeError),
    (torch.float32, "cpu", TypeError), (torch.float32, "short", ValueError)])
def test_fused_objective_refuses_what_the_kernels_cannot_read(vol, ref, error, lin_filters):
    """Types, devices and shapes of the fused operation's inputs, refused
    before their pointers are used."""
    shape = (5, 6, 8)
    v = torch.zeros((1,) + shape, device="cuda", dtype=vol)
    q = torch.zeros((1, 3) + shape + (2,), device="cpu" if ref == "cpu" else "cuda")
    q = q[:, :2] if ref == "short" else q.to(ref) if isinstance(ref, torch.dtype) else q
    with pytest.raises(error):
        AG.FilterSsd.apply(v, lin_filters, q)


@pytest.mark.parametrize("unpack", [lambda t: t.movedim(1, -1).contiguous().movedim(-1, 1), lambda t: t.double()])
def test_fused_objective_under_saved_tensor_hooks(unpack, lin_filters):
    """A saved-tensor hook that gives the residual back with other strides, or
    in float64, changes neither gradient of the fused operation."""
    m, q, _ = _objective_inputs((5, 6, 8), 6, lin_filters)
    grads = []
    for hook in (lambda t: t, unpack):
        v = m[None].clone().requires_grad_(True)
        r = q.clone().requires_grad_(True)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), hook):
            loss = AG.FilterSsd.apply(v, lin_filters, r)
        grads.append(torch.autograd.grad(loss, (v, r)))
    for a, b in zip(*grads):
        assert torch.equal(a, b)
