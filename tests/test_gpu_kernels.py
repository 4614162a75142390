"""Kernel-level parity of the CUDA path (through the C-ABI) with the oracle
and with the golden fixtures made by the reference's own kernels.

Tolerance (FP32 parity, the reference's 1e-4 relative): for every volume
output, max |gpu - ref| <= 1e-4 * max |ref| (norm-wise relative error)."""
import numpy as np
import pytest
import torch

from conftest import rel_err
from broccoli_b200 import _lib as L
from broccoli_b200 import filters as F
from broccoli_b200.api import Context

pytestmark = pytest.mark.gpu
TOL = 1e-4


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def test_filter_matches_golden(ctx, golden, lin_filters):
    q = ctx.filter3d(cuda(np.stack([golden["base"], golden["moved"]])), lin_filters).cpu().numpy()
    assert rel_err(q[0], golden["q1"]) < TOL
    assert rel_err(q[1], golden["q2"]) < TOL


@pytest.mark.parametrize("shape", [(5, 17, 33), (11, 9, 7), (9, 40, 65), (33, 64, 64), (4, 3, 2)])
@pytest.mark.parametrize("nf", [3, 6])
@pytest.mark.parametrize("prec", [L.PREC_FP32, L.PREC_FP32_GENERAL])
def test_filter_odd_shapes_vs_oracle(ctx, orc, bank, shape, nf, prec):
    """FP32 (even/odd half-tap kernel for these quadrature banks) and
    FP32_GENERAL (all 343 taps) against the oracle."""
    rng = np.random.default_rng(sum(shape) + nf)
    vol = (rng.standard_normal(shape) * 50 + 100).astype(np.float32)
    flt = bank["linear"] if nf == 3 else bank["nonlinear"]
    ref = orc.filter3d(vol, flt)
    got = ctx.filter3d(cuda(vol), flt, precision=prec).cpu().numpy()[0]
    assert got.shape == ref.shape
    assert rel_err(got, ref) < TOL


@pytest.mark.parametrize("nf", [3, 6])
def test_filter_non_symmetric_bank(ctx, orc, nf):
    """A bank without even/odd symmetry takes the general kernel."""
    rng = np.random.default_rng(40 + nf)
    flt = rng.standard_normal((nf, 2, 7, 7, 7)).astype(np.float32)
    vol = rng.standard_normal((12, 20, 36)).astype(np.float32)
    ref = orc.filter3d(vol, flt)
    got = ctx.filter3d(cuda(vol), flt).cpu().numpy()[0]
    assert rel_err(got, ref) < TOL


def test_filter_batch_matches_single(ctx, lin_filters):
    rng = np.random.default_rng(5)
    vols = rng.standard_normal((4, 9, 12, 20)).astype(np.float32)
    qb = ctx.filter3d(cuda(vols), lin_filters).cpu().numpy()
    for b in range(4):
        qs = ctx.filter3d(cuda(vols[b]), lin_filters).cpu().numpy()[0]
        assert np.array_equal(qb[b], qs)


def test_lognormal_filters_are_quadrature(ctx):
    flt = F.linear_registration_filters()
    # a plane wave along x: filter 0 responds with a constant-magnitude
    # analytic signal, the other two barely respond.
    x = np.arange(40)
    vol = np.broadcast_to(np.cos(np.pi / 3 * x), (20, 24, 40)).astype(np.float32)
    q = ctx.filter3d(cuda(vol), flt).cpu().numpy()[0]
    inner = q[:, 8:-8, 8:-8, 8:-8]
    mag = np.abs(inner[0])
    assert mag.std() / mag.mean() < 0.05
    assert np.abs(inner[1]).mean() < 0.05 * mag.mean()


def test_normal_equations_match_golden(ctx, golden):
    q1 = torch.from_numpy(golden["q1"]).cuda()
    q2 = torch.from_numpy(golden["q2"]).cuda()
    A, h = ctx.normal_equations(q1, q2[None])
    A = A.cpu().numpy()[0]
    h = h.cpu().numpy()[0]
    assert rel_err(A, golden["A"]) < TOL
    assert rel_err(h, golden["h"]) < TOL
    # zero structure identical
    assert np.array_equal(A != 0, golden["A"] != 0)


def test_solve_matches_golden(ctx, golden):
    A = torch.from_numpy(golden["A"].astype(np.float64)).cuda()
    h = torch.from_numpy(golden["h"].astype(np.float64)).cuda()
    p = ctx.solve(A, h).cpu().numpy()[0]
    np.testing.assert_allclose(p, golden["p_solve"], rtol=1e-6, atol=1e-7)


def test_solve_zero_system(ctx):
    A = torch.zeros((2, 12, 12), dtype=torch.float64, device="cuda")
    h = torch.zeros((2, 12), dtype=torch.float64, device="cuda")
    p = ctx.solve(A, h).cpu().numpy()
    assert np.all(p == 0)


def test_warp_affine_matches_golden(ctx, golden):
    out = ctx.warp_affine(cuda(golden["moved"]), torch.from_numpy(golden["p_solve"]).cuda())
    assert rel_err(out.cpu().numpy()[0], golden["warp_affine"]) < TOL


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 7, 9), (2, 8, 32), (3, 33, 31), (5, 1, 1), (33, 64, 64), (6, 9, 65),
                                   (148, 8, 63), (49, 50, 70), (3, 97, 165), (1, 120, 300)])
def test_warp_affine_pairs_of_planes(ctx, shape):
    """Odd and single planes, ragged tiles, positions on every side of the
    volume, and positions no 32-bit index holds, against the clamped trilinear
    sample in FP64."""
    D, H, W = shape
    g = torch.Generator().manual_seed(7)
    vol = torch.randn((4, D, H, W), generator=g)
    p = torch.randn((4, 12), generator=g) * 0.02
    p[:, :3] *= 100.0
    p[2, :3] = torch.tensor([1e7, -1e7, 0.25])
    p[3, :3] = torch.tensor([-0.5, 3e9, -3e9])
    out = ctx.warp_affine(vol.cuda(), p.cuda()).cpu().double()
    z, y, x = torch.meshgrid(*[torch.arange(n, dtype=torch.float64) for n in shape], indexing="ij")
    rel = [c - (n - 1) / 2 for c, n in ((x, W), (y, H), (z, D))]
    for b in range(4):
        q = p[b].double()
        lo, hi, fr = [], [], []
        for k, (c, n) in enumerate(((x, W), (y, H), (z, D))):
            pos = c + q[k] + sum(q[3 + 3 * k + j] * rel[j] for j in range(3))
            f = pos.floor()
            lo.append(f.clamp(0, n - 1).long())
            hi.append((f + 1).clamp(0, n - 1).long())
            fr.append(pos - f)
        ref = torch.zeros(shape, dtype=torch.float64)
        for corner in range(8):
            i = [hi[k] if corner >> k & 1 else lo[k] for k in range(3)]
            w = [fr[k] if corner >> k & 1 else 1 - fr[k] for k in range(3)]
            ref += w[0] * w[1] * w[2] * vol[b].double()[i[2], i[1], i[0]]
        # a position takes six roundings of at most half a step of its
        # magnitude (below 128: 2^-18); the sample's slope along an axis is at
        # most twice the largest value
        half = 2.0 ** (np.ceil(np.log2(1.2 * max(shape) + 16)) - 25)
        tol = (3 * 2 * 6 * half + 8 * 2.0**-23) * float(vol.abs().max())
        assert (out[b] - ref).abs().max() <= tol


@pytest.mark.parametrize("shape", [(3, 5, 7), (4, 9, 33), (2, 8, 65), (5, 64, 64)])
@pytest.mark.parametrize("far", [0.4, 5e6, -3e9, float("inf"), float("nan")])
def test_warp_field_lanes_of_a_warp_mixed(ctx, shape, far):
    """Lanes of one warp whose positions are inside, outside, beyond the small
    floor, infinite or NaN, in a random mixture (and warps with lanes past the
    volume's end), give what a field of one kind alone gives at each voxel."""
    g = torch.Generator().manual_seed(sum(shape))
    vol = torch.randn(shape, generator=g).cuda()
    near = (torch.rand((3,) + shape, generator=g) - 0.5).cuda()
    out = torch.full((3,) + shape, far, device="cuda")
    pick = (torch.rand(shape, generator=g) < 0.5).cuda()
    mixed = torch.where(pick, near, out)
    a, b, m = (ctx.warp_field(vol, *f) for f in (near, out, mixed))
    want = torch.where(pick, a, b)
    assert torch.equal(m.isnan(), want.isnan())
    assert torch.equal(m.nan_to_num(), want.nan_to_num())


@pytest.mark.parametrize("shape", [(1, 100, 65), (25, 17, 31), (33, 40, 64), (8, 30, 65)])
def test_warp_affine_batch_size_does_not_change_a_volume(ctx, shape):
    """A volume warped alone (one plane per thread) and among 200 (two planes)
    gives the same bits: positions inside, across the edges, far outside,
    infinite and NaN."""
    D, H, W = shape
    tiles = ((W + 31) // 32) * ((H + 7) // 8) * ((D + 1) // 2)
    assert tiles < 4 * 148 <= tiles * 16  # the launches take both forms
    g = torch.Generator().manual_seed(D)
    vol = torch.randn((8,) + shape, generator=g).cuda()
    p = torch.randn((8, 12), generator=g) * 0.05
    p[:, :3] *= 40.0
    p[4, 3], p[5, 1], p[6, 8], p[7, 2] = 2e5, 7e6, float("inf"), float("nan")
    p = p.cuda()
    many = ctx.warp_affine(vol.repeat(25, 1, 1, 1), p.repeat(25, 1))
    for k in range(8):
        one, all_k = ctx.warp_affine(vol[k:k + 1], p[k:k + 1]), many[k::8]
        assert torch.equal(all_k.isnan(), one.expand_as(all_k).isnan())
        assert torch.equal(all_k.nan_to_num(), one.expand_as(all_k).nan_to_num())


@pytest.mark.parametrize("batch", [1, 3])
def test_warp_affine_lanes_of_a_warp_mixed(ctx, batch):
    """A stretch of 2^23 along x about a central voxel: in every warp the lane
    at the centre samples it, the others lie beyond the small floor on both
    sides and take the edges.  One volume takes one plane per thread, three
    take two."""
    D, H, W = 40, 64, 65
    g = torch.Generator().manual_seed(batch)
    vol = torch.randn((batch, D, H, W), generator=g).cuda()
    p = torch.zeros((batch, 12), device="cuda")
    p[:, 3] = 2.0 ** 23
    out = ctx.warp_affine(vol, p)
    want = torch.cat([vol[..., :1].expand(-1, -1, -1, 32), vol[..., 32:33], vol[..., -1:].expand(-1, -1, -1, 32)], -1)
    assert torch.equal(out, want)


def test_warp_field_matches_golden(ctx, golden):
    out = ctx.warp_field(cuda(golden["moved"]), cuda(golden["field_x"]), cuda(golden["field_y"]),
                         cuda(golden["field_z"]))
    assert rel_err(out.cpu().numpy(), golden["warp_field"]) < TOL


def test_warp_identity_is_exact(ctx, golden):
    v = cuda(golden["moved"])
    out = ctx.warp_affine(v, torch.zeros(12, device="cuda"))
    assert torch.equal(out[0], v)


def test_smoothing_matches_golden(ctx, golden):
    fs = golden["smooth_filter"]
    out = ctx.smooth3d(cuda(golden["moved"]), fs, fs, fs).cpu().numpy()
    assert rel_err(out, golden["smooth"]) < TOL
    out = ctx.smooth3d(cuda(golden["moved"]), fs, fs, fs, cert=cuda(golden["cert"]),
                       smoothed_cert=cuda(golden["smooth_cert"])).cpu().numpy()
    assert rel_err(out, golden["smooth_normalized"]) < TOL


def test_smoothing_in_place_and_ragged_sizes(ctx, orc):
    """The fused smoothing (one kernel, z-marching) on sizes that are not
    multiples of its 32 x 8 x 32 tile, batched, against the oracle's three
    passes; and written over its own input (the output then goes through a
    temporary) with the same result."""
    import ctypes
    rng = np.random.default_rng(4)
    vols = rng.standard_normal((3, 37, 21, 45)).astype(np.float32)
    fx, fy, fz = (orc.smoothing_filter_sigma(s) for s in (1.0, 2.0, 3.0))
    got = ctx.smooth3d(cuda(vols), fx, fy, fz).cpu().numpy()
    for b in range(3):
        assert rel_err(got[b], orc.smooth3d(vols[b], fx, fy, fz)) < TOL
    v = cuda(vols)
    taps = [np.ascontiguousarray(f, np.float32) for f in (fx, fy, fz)]
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert L.lib().brc_smooth3d(ctx.handle, P(v), 45, 21, 37, 3, *[t.ctypes.data_as(ctypes.c_void_p) for t in taps],
                                None, None, P(v)) == 0
    torch.cuda.synchronize()
    assert torch.equal(v.cpu(), torch.from_numpy(got))


def test_rescale_matches_golden(ctx, golden):
    out = ctx.rescale_linear(cuda(golden["moved"]), (11, 13, 17)).cpu().numpy()
    assert rel_err(out, golden["rescale"]) < TOL


def test_smooth_normalized_matches_golden(ctx):
    """brc_smooth_normalized against the reference kernels' output: the same
    NaN voxels, the rest within 1e-4 of the largest value."""
    import os
    g = np.load(os.path.join(os.path.dirname(__file__), "golden", "smooth_normalized.npz"))
    fs = g["filter"]
    out = ctx.smooth_normalized(cuda(g["vols"]), cuda(g["mask"]), fs, fs, fs).cpu().numpy()
    ref = g["out"]
    assert np.array_equal(np.isnan(out), np.isnan(ref))
    fin = np.isfinite(ref)
    assert np.abs(out[fin] - ref[fin]).max() <= TOL * np.abs(ref[fin]).max()


@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 8, 2), (9, 9, 31), (8, 7, 32), (17, 8, 33), (9, 9, 63), (8, 7, 64), (17, 8, 65),
                                   (16, 17, 128), (33, 5, 130)])
@pytest.mark.parametrize("weighted", [False, True])
def test_smoothing_tile_edges_vs_oracle(ctx, orc, shape, weighted):
    """Sizes at the edges of the smoothing's 32 x 8 tiles, octets and groups
    of eight planes, with odd and even widths (single and paired accesses),
    plain and as the normalised smoothing, whose quotient is multiplied by
    the mask in the same kernel.  Same bar as the golden tests, 1e-4."""
    rng = np.random.default_rng(sum(shape))
    vols = rng.standard_normal((2,) + shape).astype(np.float32)
    taps = [orc.smoothing_filter_sigma(s) for s in (1.0, 2.0, 5.0)]
    if weighted:
        mask = np.where(rng.random(shape) < 0.5, 1.0, 0.001).astype(np.float32)
        sm = orc.smooth3d(mask, *taps)
        got = ctx.smooth_normalized(cuda(vols), cuda(mask), *taps).cpu().numpy()
        ref = [orc.smooth3d(v, *taps, mask, sm) * mask for v in vols]
        parts = ctx.smooth3d(cuda(vols), *taps, cert=cuda(mask), smoothed_cert=ctx.smooth3d(cuda(mask), *taps))
        assert np.array_equal(got, (parts * cuda(mask)).cpu().numpy())
    else:
        got = ctx.smooth3d(cuda(vols), *taps).cpu().numpy()
        ref = [orc.smooth3d(v, *taps) for v in vols]
    for b in range(2):
        assert rel_err(got[b], ref[b]) < TOL


def test_filter_shape_inside_a_capture(lin_filters):
    """A capture cannot time: it takes the launch shape known for the nearest
    launch size of the volume shape (powers of two, the larger of two equally
    near), and the untimed one where none is known.  One warm call outside thus
    serves captures of every batch."""
    c = Context(0)
    shape = (9, 11, 13)
    vols = torch.rand((4,) + shape, device="cuda")
    c.filter3d(vols, lin_filters)  # loads the kernels; times launches of 4
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        c.filter3d(vols, lin_filters)
        other = c.selftest_filter_shape((9, 11, 14), 4, lin_filters)
    assert other == 3  # the depth that divides 9 planes
    for known, queries in [({4: 8}, {1: 8, 3: 8, 7: 8, 200: 8}), ({1: 6}, {1: 6, 2: 8, 4: 8}),
                           ({16: 2}, {2: 8, 7: 8, 8: 2, 40: 2})]:
        for batch, shape_code in known.items():
            assert c.selftest_filter_shape(shape, batch, lin_filters, set=shape_code) == shape_code
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            c.filter3d(vols, lin_filters)
            got = {batch: c.selftest_filter_shape(shape, batch, lin_filters) for batch in queries}
        assert got == queries
    c.close()


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 5, 2), (7, 9, 4), (5, 17, 33), (9, 8, 36), (11, 20, 63)])
@pytest.mark.parametrize("nf", [3, 6])
@pytest.mark.parametrize("kind", ["symmetric", "general", "asymmetric"])
@pytest.mark.parametrize("offset", [0, 1])
def test_filter_launch_shapes_agree(ctx, bank, shape, nf, kind, offset):
    """Every launch shape of the FP32 filtering that the timing can pick, on
    widths below and off the quad, depths below the block's and volumes that
    are not 16-byte aligned: the same responses bit for bit, with nothing
    written outside them, and within the suite's 1e-4 of the FP64 convolution
    (the shape of the summation order that all share)."""
    gen = torch.Generator().manual_seed(sum(shape) + nf)
    flt = bank["linear" if nf == 3 else "nonlinear"]
    if kind == "asymmetric":
        flt = torch.randn((nf, 2, 7, 7, 7), generator=gen).numpy()
    prec = L.PREC_FP32_GENERAL if kind == "general" else L.PREC_FP32
    D, H, W = shape
    vols = torch.randn((2,) + shape, generator=gen)
    ref = torch.nn.functional.conv3d(vols.double()[:, None], torch.from_numpy(flt).double().flip(2, 3, 4).reshape(
        2 * nf, 1, 7, 7, 7), padding=3).reshape((2, nf, 2) + shape).movedim(2, -1)
    src = torch.zeros(vols.numel() + 1, device="cuda")[offset:offset + vols.numel()]
    src.copy_(vols.reshape(-1))
    f = np.ascontiguousarray(flt, np.float32)
    outs = {}
    for code in range(1, 64):
        try:
            ctx.selftest_filter_shape(shape, 2, flt, prec, set=code)
        except L.BrcError as e:
            assert e.status == L.BRC_ERR_INVALID
            continue
        buf = torch.full((ref.numel() + 64,), 7.0, device="cuda")
        assert L.lib().brc_filter3d(ctx.handle, src.data_ptr(), W, H, D, 2, W * H * D, f.ctypes.data, nf, prec,
                                    buf.data_ptr() + 128) == 0
        assert bool((buf[:32] == 7.0).all()) and bool((buf[-32:] == 7.0).all())
        outs[code] = buf[32:-32].reshape(ref.shape).cpu()
    assert len(outs) == (7 if nf == 3 else 5)
    first = next(iter(outs.values()))
    assert all(torch.equal(o, first) for o in outs.values())
    assert float((first.double() - ref).abs().max() / ref.abs().max()) < TOL
