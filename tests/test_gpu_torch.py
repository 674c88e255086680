"""The differentiable Jacobian: adjoint kernel against FP64 central finite
differences and against the reference's analytic gradient (GPU)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _affected(shape, q):
    """Voxels whose Jacobian reads voxel q (the radius-2 cross)."""
    out = []
    for a in range(3):
        for t in range(-2, 3):
            p = list(q)
            p[a] += t
            if all(0 <= p[i] < shape[i] for i in range(3)) and (a == 0 or t != 0):
                out.append(tuple(p))
    return out


def fd_check(field64, w, grad, probes, spacing=(1.0, 1.0, 1.0), h=1e-6, order=4):
    """Central differences of L = sum w J(u) at `probes` (component, z, y, x),
    differenced only over the voxels each probe affects."""
    import torch
    from disptools_b200 import torch_ops
    fd = []
    for c, z, y, x in probes:
        f = field64.clone()
        f[c, z, y, x] += h
        Jp = torch_ops.jacobian_raw(f, spacing, order)
        f[c, z, y, x] -= 2 * h
        Jm = torch_ops.jacobian_raw(f, spacing, order)
        idx = _affected(field64.shape[1:], (z, y, x))
        zi, yi, xi = (torch.tensor(v, device=f.device) for v in zip(*idx))
        fd.append(float(torch.sum(w[zi, yi, xi] * (Jp[zi, yi, xi] - Jm[zi, yi, xi]))) / (2 * h))
    got = np.array([float(grad[c, z, y, x]) for c, z, y, x in probes])
    return got, np.array(fd)


@pytest.mark.parametrize("shape", [(14, 12, 10), (13, 11, 19)])
def test_adjoint_fp64_vs_finite_differences(shape):
    """The second shape has odd extents and a deep interior along x, where
    the gather uses its constant weights."""
    import torch
    from disptools_b200 import torch_ops
    from disptools_b200.synthetic import smooth_field
    f = torch.from_numpy(smooth_field(shape, sigma=2.0, max_disp=0.8, seed=1)).cuda()
    f.requires_grad_(True)
    rng = np.random.default_rng(2)
    w = torch.from_numpy(rng.standard_normal(shape)).cuda()
    sp = (0.9, 1.1, 1.3)
    J = torch_ops.jacobian(f, sp)
    (J * w).sum().backward()
    probes = [(int(c), int(z), int(y), int(x)) for c, z, y, x in
              zip(rng.integers(0, 3, 300), rng.integers(0, shape[0], 300), rng.integers(0, shape[1], 300),
                  rng.integers(0, shape[2], 300))]
    got, fd = fd_check(f.detach(), w, f.grad, probes, sp)
    np.testing.assert_allclose(got, fd, rtol=1e-6, atol=1e-7)


@pytest.mark.parametrize("shape", [(21, 40, 68), (96, 112, 100)])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_adjoint_tma_and_plain_paths_agree(dtype, shape):
    """The TMA passes (aligned field: weight pass on the TMA stencil kernel,
    TMA gather) and the plain-load passes (a field 8 bytes off a 16-byte
    boundary) give the same gradient on every voxel: several tiles per axis,
    tiles on every face (the gather's x-face and general paths) and a deep
    interior (its fourth-order path); bit for bit in FP64."""
    import torch
    from disptools_b200 import torch_ops
    from disptools_b200.synthetic import smooth_field
    tdt = getattr(torch, dtype)
    f = torch.from_numpy(smooth_field(shape, sigma=3.0, max_disp=1.5, seed=4)).to(tdt).cuda()
    rng = np.random.default_rng(5)
    w = torch.from_numpy(rng.standard_normal(shape)).to(tdt).cuda()
    sp = (0.9, 1.2, 1.05)
    g_tma = torch_ops.jacobian_adjoint_raw(f, w, sp)
    k = 8 // f.element_size()  # elements in 8 bytes
    buf = torch.zeros(f.numel() + k, dtype=tdt, device="cuda")
    buf[k:] = f.reshape(-1)
    off = buf[k:].view(f.shape)
    assert off.data_ptr() % 16 == 8
    g_plain = torch_ops.jacobian_adjoint_raw(off, w, sp)
    if dtype == "float64":
        torch.testing.assert_close(g_tma, g_plain, rtol=0, atol=0)
    else:
        torch.testing.assert_close(g_tma, g_plain, rtol=1e-5, atol=1e-5)


def test_adjoint_matches_reference_gradient(oracle_pd2):
    """With second-order differences the cost gradient of the reference
    (src/displacement_field_gradient.c:26-145) is the adjoint applied to
    2 e' (e' the regularised error), on voxels away from the boundary."""
    import torch
    from disptools_b200 import torch_ops
    from disptools_b200.synthetic import smooth_field
    shape = (16, 15, 14)
    f = smooth_field(shape, sigma=2.0, max_disp=1.5, seed=3)
    rng = np.random.default_rng(4)
    Jt = 1.0 + 0.1 * rng.standard_normal(shape)
    mask = rng.random(shape) < 0.5
    sp = (1.0, 1.2, 0.8)
    delta, zeta = 0.9, 10.0  # a delta above some J values exercises the regulariser
    J2 = oracle_pd2.jacobian(f, sp)
    _, _, v = oracle_pd2.compute_error(Jt, J2, mask, 0.2)
    g_ref, _ = oracle_pd2.gradient(f, J2, v, delta, zeta, sp)
    ep = v + np.where(J2 < delta, zeta * (J2 - delta), 0.0)
    g = torch_ops.jacobian_adjoint_raw(torch.from_numpy(f).cuda(), torch.from_numpy(2 * ep).cuda(),
                                       sp, order=2).cpu().numpy()
    inner = (slice(None),) + (slice(3, -3),) * 3
    np.testing.assert_allclose(g[inner], g_ref[inner], rtol=1e-10, atol=1e-12)


def test_batched_fp32_autograd_config3():
    """4 fields of 192x224x192 (smooth noise, sigma 6, max |u| = 3): FP32
    forward and backward; the backward checked on 1000 random voxels against
    FP64 central differences (h = 1e-6)."""
    import torch
    from disptools_b200 import torch_ops
    from disptools_b200.synthetic import smooth_field
    shape = (192, 224, 192)
    fields = np.stack([smooth_field(shape, 6.0, 3.0, seed=s) for s in range(4)])
    f32 = torch.from_numpy(fields).float().cuda().requires_grad_(True)
    rng = np.random.default_rng(9)
    w = torch.from_numpy(rng.standard_normal((4,) + shape)).cuda()
    J = torch_ops.jacobian(f32)
    assert J.shape == (4,) + shape
    (J * w.float()).sum().backward()
    g = f32.grad
    errs = []
    for b in range(4):
        f64 = torch.from_numpy(fields[b]).cuda()
        probes = [(int(c), int(z), int(y), int(x)) for c, z, y, x in
                  zip(rng.integers(0, 3, 250), rng.integers(0, shape[0], 250),
                      rng.integers(0, shape[1], 250), rng.integers(0, shape[2], 250))]
        got, fd = fd_check(f64, w[b], g[b], probes)
        scale = np.maximum(np.abs(fd), 1.0)
        errs.append(np.max(np.abs(got - fd) / scale))
    assert max(errs) <= 1e-4, errs


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("shape", [(3, 3, 4), (5, 9, 12), (7, 17, 36), (40, 40, 96), (37, 21, 100),
                                   (30, 53, 132)])
def test_fused_adjoint_equals_two_pass(monkeypatch, dtype, shape):
    """The fused adjoint kernel (one launch, weights on chip,
    DISPTOOLS_B200_ADJOINT=fused) against the weight pass + gather: bit for bit in
    FP64, to float rounding in FP32.  The shapes give partial tiles on every
    axis, volumes of 3 voxels, and (40 x 40 x 96) tiles whose every voxel is
    four cells from the faces (the constant-weight path)."""
    import torch

    import disptools_b200 as dt
    from disptools_b200 import torch_ops
    from disptools_b200.synthetic import smooth_field
    t = getattr(torch, dtype)
    f = torch.from_numpy(smooth_field(shape, sigma=2.0, max_disp=0.8, seed=3)).to(t).cuda()
    w = torch.from_numpy(np.random.default_rng(4).standard_normal(shape)).to(t).cuda()
    sp = (0.9, 1.1, 1.3)
    monkeypatch.setenv("DISPTOOLS_B200_ADJOINT", "fused")
    n0 = dt.kernel_launch_count()
    fused = torch_ops.jacobian_adjoint_raw(f, w, sp)
    torch.cuda.synchronize()
    assert dt.kernel_launch_count() - n0 == 1  # one kernel: the fused path ran
    monkeypatch.delenv("DISPTOOLS_B200_ADJOINT")
    n0 = dt.kernel_launch_count()
    two = torch_ops.jacobian_adjoint_raw(f, w, sp)
    torch.cuda.synchronize()
    assert dt.kernel_launch_count() - n0 == 2
    a, b = fused.cpu().numpy(), two.cpu().numpy()
    if dtype == "float64":
        np.testing.assert_array_equal(a, b)
    else:
        np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6 * np.abs(b).max())


@pytest.mark.parametrize("shape", [(3, 3, 4), (7, 17, 36), (21, 40, 68), (40, 40, 96), (30, 53, 132)])
def test_autograd_cofactor_path_matches_weight_path(monkeypatch, shape):
    """The FP32 autograd forward that keeps C = cof * ih and the one-gather
    backward (the default for TMA-friendly layouts) against the weight pass +
    gather (DISPTOOLS_B200_AUTOGRAD=weights): the same map bit for bit, the
    same gradient to float rounding (grad_J * (cof * ih) against
    (grad_J * cof) * ih); single and batched fields."""
    import torch
    from disptools_b200 import torch_ops
    from disptools_b200.synthetic import smooth_field
    fields = np.stack([smooth_field(shape, sigma=2.0, max_disp=0.8, seed=s) for s in (3, 4)])
    w = torch.from_numpy(np.random.default_rng(5).standard_normal((2,) + shape)).float().cuda()
    sp = (0.9, 1.1, 1.3)

    def run(batched):
        f = torch.from_numpy(fields).float().cuda().requires_grad_(True)
        if batched:
            J = torch_ops.jacobian(f, sp)
            (J * w).sum().backward()
        else:
            J = torch.stack([torch_ops.jacobian(f[b], sp) for b in range(2)])
            (J * w).sum().backward()
        return J.detach(), f.grad

    assert torch_ops.cof_supported(torch.zeros((3,) + shape, device="cuda"))
    for batched in (False, True):
        Jc, gc = run(batched)
        monkeypatch.setenv("DISPTOOLS_B200_AUTOGRAD", "weights")
        Jw, gw = run(batched)
        monkeypatch.delenv("DISPTOOLS_B200_AUTOGRAD")
        torch.testing.assert_close(Jc, Jw, rtol=0, atol=0)
        scale = gw.abs().max().item()
        torch.testing.assert_close(gc, gw, rtol=1e-5, atol=1e-6 * scale)


def test_autograd_cofactor_path_unsupported_layouts_fall_back():
    """Widths that are not a multiple of four float32 elements and float64
    fields take the weight pass + gather."""
    import torch
    from disptools_b200 import torch_ops
    assert not torch_ops.cof_supported(torch.zeros((3, 8, 8, 9), device="cuda"))
    assert not torch_ops.cof_supported(torch.zeros((3, 8, 8, 8), dtype=torch.float64, device="cuda"))
    f = torch.rand((3, 8, 8, 9), device="cuda", requires_grad=True)
    torch_ops.jacobian(f).sum().backward()
    assert f.grad is not None and torch.isfinite(f.grad).all()


def test_cof_entry_points_reject_unsupported_layouts():
    """The C entry points of the cofactor path refuse layouts their tensor
    maps cannot cover (rows not a multiple of 16 bytes, misaligned bases)
    with DTB_ERR_ARGUMENT and the error state set, and do no device work."""
    import torch
    from disptools_b200 import _native as N
    f = torch.zeros((3, 8, 8, 9), device="cuda")
    J = torch.zeros((8, 8, 9), device="cuda")
    C = torch.zeros((9, 8, 8, 9), device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    rc = N.lib.dtb_jacobian_cof_device(N.PRECISION_MIXED, 9, 8, 8, 1.0, 1.0, 1.0, f.data_ptr(), J.data_ptr(),
                                       C.data_ptr(), s)
    assert rc == -1 and N.lib.disptools_has_error()
    buf = torch.zeros(9 * 8 * 8 * 8 + 1, device="cuda")
    C8 = buf[1:]  # 4 bytes off the allocation's alignment
    gJ = torch.zeros((8, 8, 8), device="cuda")
    g = torch.zeros((3, 8, 8, 8), device="cuda")
    rc = N.lib.dtb_jacobian_adjoint_cof_device(N.PRECISION_MIXED, 8, 8, 8, 1.0, 1.0, 1.0, C8.data_ptr(),
                                               gJ.data_ptr(), g.data_ptr(), s)
    assert rc == -1 and N.lib.disptools_has_error()
    N.lib.disptools_clear_error()


@pytest.mark.parametrize("shape", [(3, 5, 3), (6, 18, 33), (34, 17, 35), (5, 16, 67)])
@pytest.mark.parametrize("order", [4, 2])
def test_adjoint_of_odd_widths(oracle, oracle_pd2, shape, order):
    """Padded weights and unpaired stores: <w, dJ[v]> = <adj w, v> with the
    directional derivative of the oracle's (cubic) map by central differences,
    whose only error is h^2 det(grad v) ~ 1e-8 and rounding / h ~ 1e-12."""
    import torch
    from disptools_b200 import torch_ops
    rng = np.random.default_rng(sum(shape) + order)
    u, v = rng.normal(scale=0.2, size=(2, 3) + shape)
    w = rng.standard_normal(shape)
    sp = (0.9, 1.1, 1.3)
    o = oracle if order == 4 else oracle_pd2
    h = 1e-4
    dJ = (o.jacobian(u + h * v, sp) - o.jacobian(u - h * v, sp)) / (2 * h)
    scale = np.sum(np.abs(w * dJ))
    for dtype, tol in ((torch.float64, 1e-7), (torch.float32, 1e-5)):
        g = torch_ops.jacobian_adjoint_raw(torch.from_numpy(u).to(dtype).cuda(), torch.from_numpy(w).to(dtype).cuda(),
                                           sp, order).double().cpu().numpy()
        assert abs(np.sum(g * v) - np.sum(w * dJ)) <= tol * scale


@pytest.mark.parametrize("shape", [(3, 3, 12), (4, 6, 13), (3, 40, 16), (70, 3, 33), (8, 9, 11), (9, 7, 64)])
def test_adjoint_taps_near_faces(oracle, oracle_pd2, shape):
    """Volumes in which most taps choose a scheme, on both sides of the widths
    that stream their weights."""
    test_adjoint_of_odd_widths(oracle, oracle_pd2, shape, 4)


@pytest.mark.parametrize("shape", [(12, 20, 48), (12, 20, 45)])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_adjoint_keeps_infinities_local(shape, value):
    """A weight that is not finite reaches the voxels that have a tap on it
    (those that a large finite one changes) and no others, with or without
    the saved cofactors."""
    import torch
    from disptools_b200 import torch_ops
    rng = np.random.default_rng(3)
    u = rng.normal(scale=0.2, size=(3,) + shape)
    w = rng.standard_normal(shape)

    def through_autograd(field, weight):
        leaf = field.clone().requires_grad_(True)
        return torch.autograd.grad(torch_ops.jacobian(leaf), leaf, weight)[0]

    for dtype in (torch.float32, torch.float64):
        field, weight = torch.from_numpy(u).to(dtype).cuda(), torch.from_numpy(w).to(dtype).cuda()
        for adjoint in (torch_ops.jacobian_adjoint_raw, through_autograd):
            for place in ((0, 0, 0), (1, 10, 31), (6, 1, 32), (6, 10, 1), (6, 10, 20), (11, 19, shape[2] - 2)):
                results = []
                for v in (0.0, 1e30, value):
                    weight[place] = v
                    results.append(adjoint(field, weight))
                zero, large, bad = results
                reached = large != zero
                assert torch.equal(~torch.isfinite(bad), reached)
                assert torch.equal(bad[~reached], zero[~reached])
                weight[place] = float(w[place])


def test_adjoint_under_a_memory_limit():
    """Odd widths pad their weights only where a memory limit has room for it:
    20 x 21 x 45 needs 682240 bytes dense and 726016 padded."""
    import torch

    import disptools_b200 as dt
    from disptools_b200 import _native as N
    from disptools_b200 import torch_ops
    rng = np.random.default_rng(5)
    shape = (20, 21, 45)
    field = torch.from_numpy(rng.normal(scale=0.2, size=(3,) + shape)).float().cuda()
    weight = torch.from_numpy(rng.standard_normal(shape)).float().cuda()
    want = torch_ops.jacobian_adjoint_raw(field, weight)
    try:
        N.check(N.lib.dtb_set_device_memory_limit(700000))
        got = torch_ops.jacobian_adjoint_raw(field, weight)
        N.check(N.lib.dtb_set_device_memory_limit(682239))
        with pytest.raises(dt.DisptoolsError):
            torch_ops.jacobian_adjoint_raw(field, weight)
    finally:
        N.check(N.lib.dtb_set_device_memory_limit(0))
    # Thirteen terms a component, each rounded once in either order.
    assert float((got - want).abs().max()) <= 13 * 2 ** -24 * 13 * float(want.abs().max())


def test_backward_on_a_thread_without_a_context():
    """The backward of a fresh process, its gradient's memory cached: the first
    device work of the autograd thread."""
    import subprocess
    import sys
    code = ("import torch\n"
            "from disptools_b200 import torch_ops\n"
            "f = 0.1 * torch.randn(3, 40, 40, 40, device='cuda')\n"
            "w = torch.randn(40, 40, 40, device='cuda')\n"
            "spare = [torch.empty_like(f) for _ in range(8)]\n"
            "del spare\n"
            "f.requires_grad_(True)\n"
            "J = torch_ops.jacobian(f)\n"
            "torch.autograd.grad(J, f, w)\n"
            "torch.cuda.synchronize()\n")
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300)


@pytest.mark.parametrize("shape, order, weights, gather", [
    ((6, 18, 33), 2, "k_adjoint_w", "k_adjoint_gather"),
    ((130, 97, 99), 2, "k_jacobian_async", "k_adjoint_gather"),
    ((300, 3, 3), 4, "k_adjoint_w", "k_adjoint_gather"),
    ((40, 41, 3), 4, "k_adjoint_w", "k_adjoint_gather"),
    ((30, 3, 71), 4, "k_adjoint_w", "k_adjoint_gather"),
    ((50, 16, 63), 4, "k_jacobian_async", "k_gather_tma"),
    ((20, 64, 7), 4, "k_jacobian_async", "k_adjoint_gather"),
])
def test_adjoint_by_tiles_or_by_voxels(oracle, oracle_pd2, shape, order, weights, gather):
    """Small volumes of second order and those that leave a tile mostly idle
    take their weights with a thread per voxel (up to three times as fast
    there), low ones their gather by plain loads; the identity and tolerances of
    test_adjoint_of_odd_widths hold for each."""
    import torch
    from disptools_b200 import torch_ops
    from tests.helpers import kernels_of
    rng = np.random.default_rng(sum(shape) + order)
    u, v = rng.normal(scale=0.2, size=(2, 3) + shape)
    w = rng.standard_normal(shape)
    sp = (0.9, 1.1, 1.3)
    o = oracle if order == 4 else oracle_pd2
    h = 1e-4
    dJ = (o.jacobian(u + h * v, sp) - o.jacobian(u - h * v, sp)) / (2 * h)
    scale = np.sum(np.abs(w * dJ))
    for dtype, tol in ((torch.float64, 1e-7), (torch.float32, 1e-5)):
        ud, wd = torch.from_numpy(u).to(dtype).cuda(), torch.from_numpy(w).to(dtype).cuda()
        g, names = kernels_of(lambda: torch_ops.jacobian_adjoint_raw(ud, wd, sp, order), weights, gather)
        assert weights in names and gather in names
        assert abs(np.sum(g.double().cpu().numpy() * v) - np.sum(w * dJ)) <= tol * scale


def _off_by_one_element(t):
    import torch
    view = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("dtype, shape", [("float64", (193, 197, 198)), ("float32", (37, 39, 68))])
def test_tma_and_element_wise_stencils_agree(dtype, shape):
    """Map and weights by the TMA kernel and, for a field off a 16-byte
    boundary, by the element-wise one, on a size that takes both and has
    partial tiles along every axis.  FP64 rounds alike; FP32 sums a derivative's
    two terms, four products a minor and three a determinant in other orders."""
    import torch
    from disptools_b200 import torch_ops
    from tests.helpers import kernels_of
    tdt = getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(7)
    f = 0.1 * torch.randn((3,) + shape, dtype=tdt, device="cuda", generator=g)
    w = torch.randn(shape, dtype=tdt, device="cuda", generator=g)
    off = _off_by_one_element(f)
    sp = (0.9, 1.2, 1.05)
    for call in (lambda u: torch_ops.jacobian_raw(u, sp), lambda u: torch_ops.jacobian_adjoint_raw(u, w, sp)):
        tma, names = kernels_of(lambda: call(f), "k_jacobian_tma")
        assert "k_jacobian_tma" in names and "k_jacobian_async" not in names
        plain, names = kernels_of(lambda: call(off), "k_jacobian_async")
        assert "k_jacobian_async" in names and "k_jacobian_tma" not in names
        if dtype == "float64":
            torch.testing.assert_close(tma, plain, rtol=0, atol=0)
        else:
            torch.testing.assert_close(tma, plain, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("shape", [(20, 21, 45), (5, 31, 13), (9, 16, 67), (35, 17, 99)])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_streamed_and_plain_gathers_agree(dtype, shape):
    """The gather by TMA and, where a memory limit has no room for padded rows,
    by plain loads, from the same weights: equal in FP64, and in FP32 thirteen
    terms a component, each rounded once in either order."""
    import torch
    from disptools_b200 import _native as N
    from disptools_b200 import torch_ops
    from tests.helpers import kernels_of
    tdt = getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(8)
    f = 0.2 * torch.randn((3,) + shape, dtype=tdt, device="cuda", generator=g)
    w = torch.randn(shape, dtype=tdt, device="cuda", generator=g)
    streamed, names = kernels_of(lambda: torch_ops.jacobian_adjoint_raw(f, w), "k_gather_tma")
    assert "k_gather_tma" in names and "k_adjoint_gather" not in names
    n = int(np.prod(shape))
    try:
        N.check(N.lib.dtb_set_device_memory_limit(9 * ((n + 63) // 64 * 64) * f.element_size() + 256))
        plain, names = kernels_of(lambda: torch_ops.jacobian_adjoint_raw(f, w), "k_adjoint_gather")
    finally:
        N.check(N.lib.dtb_set_device_memory_limit(0))
    assert "k_adjoint_gather" in names and "k_gather_tma" not in names
    if dtype == "float64":
        torch.testing.assert_close(streamed, plain, rtol=0, atol=0)
    else:
        assert float((streamed - plain).abs().max()) <= 13 * 2 ** -24 * 13 * float(plain.abs().max())
