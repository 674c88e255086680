"""Jacobian kernels against the oracle and the golden vectors (GPU)."""
from __future__ import annotations

import numpy as np
import pytest

import disptools_b200 as dt

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.max(np.abs(a - b) / np.maximum(np.abs(b), 1.0)))


def test_fp64_golden_vectors_bit_exact(golden):
    g = golden["jacobian"]
    np.testing.assert_array_equal(dt.jacobian(g["sin10_field"]), g["sin10_J"])
    np.testing.assert_array_equal(dt.jacobian(g["i2_field"], (2.0, 3.0, 4.0)), g["i2_J"])
    for k in range(4):
        f, sp = g[f"rand{k}_field"], tuple(g[f"rand{k}_spacing"])
        assert rel_err(dt.jacobian(f, sp), g[f"rand{k}_J"]) <= 1e-12


@pytest.mark.parametrize("shape", [(3, 3, 3), (3, 40, 5), (9, 33, 70), (64, 64, 64),
                                   (5, 130, 17), (37, 8, 31), (4, 4, 200)])
def test_fp64_shapes_vs_oracle(oracle, shape):
    rng = np.random.default_rng(sum(shape))
    f = rng.normal(scale=0.2, size=(3,) + shape)
    sp = tuple(rng.uniform(0.5, 2.0, 3))
    assert rel_err(dt.jacobian(f, sp), oracle.jacobian(f, sp)) <= 1e-12


def _torch():
    import torch
    return torch


@pytest.mark.parametrize("order", [4, 2])
def test_device_entry_fp32_and_fp64(oracle, oracle_pd2, order):
    torch = _torch()
    from disptools_b200 import torch_ops
    o = oracle if order == 4 else oracle_pd2
    rng = np.random.default_rng(3)
    f = rng.normal(scale=0.2, size=(3, 21, 34, 45))
    sp = (0.9, 1.2, 1.05)
    ref = o.jacobian(f, sp)
    J64 = torch_ops.jacobian_raw(torch.from_numpy(f).cuda(), sp, order).cpu().numpy()
    assert rel_err(J64, ref) <= 1e-12
    J32 = torch_ops.jacobian_raw(torch.from_numpy(f).float().cuda(), sp, order).cpu().numpy()
    assert rel_err(J32.astype(np.float64), ref) <= 2e-5


@pytest.mark.parametrize("shape", [(37, 45, 68), (70, 18, 36), (3, 3, 4), (33, 17, 132), (5, 40, 8)])
def test_device_entry_tma_layouts(oracle, shape):
    """Rows a multiple of 16 bytes long take the TMA kernel: several tiles
    along every axis, partial tiles, thin volumes; FP64 to the last bits."""
    torch = _torch()
    from disptools_b200 import torch_ops
    rng = np.random.default_rng(sum(shape))
    f = rng.normal(scale=0.2, size=(3,) + shape)
    sp = tuple(rng.uniform(0.5, 2.0, 3))
    ref = oracle.jacobian(f, sp)
    J64 = torch_ops.jacobian_raw(torch.from_numpy(f).cuda(), sp).cpu().numpy()
    assert rel_err(J64, ref) <= 1e-12
    J32 = torch_ops.jacobian_raw(torch.from_numpy(f).float().cuda(), sp).cpu().numpy()
    assert rel_err(J32.astype(np.float64), ref) <= 2e-5


def test_device_entry_unaligned_field_takes_plain_kernel(oracle):
    """A field that starts off a 16-byte boundary goes to the plain-load
    kernel and gives the same map."""
    torch = _torch()
    from disptools_b200 import torch_ops
    shape = (9, 20, 24)
    rng = np.random.default_rng(7)
    f = rng.normal(scale=0.2, size=(3,) + shape)
    ref = oracle.jacobian(f)
    n = f.size
    buf = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    buf[1:] = torch.from_numpy(f.ravel()).cuda()
    view = buf[1:].view((3,) + shape)  # 8 bytes past the allocation's start
    assert view.data_ptr() % 16 == 8
    J = torch_ops.jacobian_raw(view).cpu().numpy()
    assert rel_err(J, ref) <= 1e-12
    np.testing.assert_array_equal(J, torch_ops.jacobian_raw(view.clone()).cpu().numpy())


def test_full_size_256_vs_oracle(oracle):
    torch = _torch()
    from disptools_b200 import torch_ops
    from disptools_b200.synthetic import smooth_field
    f = smooth_field((256, 256, 256), sigma=6.0, max_disp=3.0, seed=5)
    ref = oracle.jacobian(f)
    J64 = torch_ops.jacobian_raw(torch.from_numpy(f).cuda()).cpu().numpy()
    assert rel_err(J64, ref) <= 1e-12
    J32 = torch_ops.jacobian_raw(torch.from_numpy(f).float().cuda()).cpu().numpy()
    assert rel_err(J32.astype(np.float64), ref) <= 1e-4


def test_regularise():
    rng = np.random.default_rng(0)
    J = rng.random((20, 21, 22)) + 0.05
    m = rng.integers(5, size=J.shape) % 4 == 0
    P = J.copy()
    P[m] = 0.05 - rng.random()
    R = dt.regularise(P, 0.05)
    assert np.array_equal(R[~m], J[~m])
    assert np.all(R[m] == 0.05)


def test_extension_jacobian_matches(golden):
    from disptools_b200 import _disptools
    g = golden["jacobian"]
    out = np.zeros((10, 10, 10))
    _disptools.jacobian((1.0, 1.0, 1.0), g["sin10_field"], out)
    np.testing.assert_array_equal(out, g["sin10_J"])


@pytest.mark.parametrize("order", [4, 2])
@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 7, 33), (33, 8, 31), (5, 9, 65), (70, 17, 45), (2 * 32 + 3, 25, 99)])
def test_any_layout_kernel_at_tile_edges(oracle, oracle_pd2, shape, order):
    """The element-wise kernel (odd widths; a base off a 16-byte boundary;
    second order) around its 32 x 8 tiles: FP64 to 1e-12 of the oracle, FP32
    to 2e-5, and the same bits whatever the base."""
    torch = _torch()
    from disptools_b200 import torch_ops
    rng = np.random.default_rng(sum(shape))
    f = rng.normal(scale=0.2, size=(3,) + shape)
    sp = (0.9, 1.2, 1.05)
    ref = (oracle if order == 4 else oracle_pd2).jacobian(f, sp)
    for dtype, tol in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
        fd = torch.from_numpy(f).to(dtype).cuda()
        J = torch_ops.jacobian_raw(fd, sp, order)
        assert rel_err(J.double().cpu().numpy(), ref) <= tol
        off = torch.empty(fd.numel() + 1, dtype=dtype, device="cuda")[1:].view(fd.shape)
        off.copy_(fd)
        J2 = torch_ops.jacobian_raw(off, sp, order)
        if shape[2] % 2:
            assert torch.equal(J, J2)
        else:
            assert rel_err(J2.double().cpu().numpy(), ref) <= tol


@pytest.mark.parametrize("shape", [(40, 5, 3), (5, 33, 8), (4, 31, 9), (9, 65, 15), (3, 34, 16), (5, 33, 17)])
@pytest.mark.parametrize("order", [4, 2])
def test_any_layout_kernel_on_narrow_volumes(oracle, oracle_pd2, shape, order):
    """The same around its 8 x 32 tiles and the width that takes them."""
    test_any_layout_kernel_at_tile_edges(oracle, oracle_pd2, shape, order)


def test_any_layout_kernel_keeps_infinities_local(oracle):
    """An infinite value reaches only the voxels whose schemes read it, also
    on the second-order outer layers."""
    torch = _torch()
    from disptools_b200 import torch_ops
    f = np.random.default_rng(4).normal(scale=0.1, size=(3, 9, 11, 13))
    f[1, 4, 5, 3] = np.inf
    with np.errstate(invalid="ignore"):
        ref = oracle.jacobian(f)
    J = torch_ops.jacobian_raw(torch.from_numpy(f).cuda()).cpu().numpy()
    np.testing.assert_array_equal(np.isfinite(J), np.isfinite(ref))


@pytest.mark.parametrize("at", [(4, 5, 3), (2, 2, 2), (8, 10, 15), (5, 1, 12)])
def test_tma_kernel_keeps_infinities_local(oracle, at):
    """The same for the TMA kernel: the outer layers share one expression with
    the fourth-order voxels, which must not read what their scheme does not."""
    torch = _torch()
    from disptools_b200 import torch_ops
    f = np.random.default_rng(4).normal(scale=0.1, size=(3, 9, 11, 16)).astype(np.float32)
    f[(1,) + at] = np.inf
    with np.errstate(invalid="ignore"):
        ref = oracle.jacobian(f.astype(np.float64))
    J = torch_ops.jacobian_raw(torch.from_numpy(f).cuda()).cpu().numpy()
    np.testing.assert_array_equal(np.isfinite(J), np.isfinite(ref))
    ok = np.isfinite(ref)
    assert np.max(np.abs(J[ok] - ref[ok])) <= 2e-5


def test_maps_of_host_arrays_on_kept_and_own_memory(oracle):
    """Maps on both sides of the 2 MiB that are kept (40^3 and 41^3), from
    threads at once, of which one has them, and after a release."""
    from concurrent.futures import ThreadPoolExecutor
    rng = np.random.default_rng(2)
    fields = [rng.normal(scale=0.2, size=(3, n, n, n)) for n in (8, 31, 32, 33, 40, 41)]
    refs = [oracle.jacobian(f) for f in fields]
    dt.release_device_memory()
    with ThreadPoolExecutor(4) as pool:
        for _ in range(3):
            for got, ref in zip(pool.map(dt.jacobian, fields * 3), refs * 3):
                np.testing.assert_allclose(got, ref, rtol=0, atol=1e-13)
            for got, ref in zip(pool.map(lambda J: dt.regularise(J, 0.9), refs * 3), refs * 3):
                np.testing.assert_array_equal(got, np.where(ref < 0.9, 0.9, ref))
    dt.release_device_memory()
    for f, ref in zip(fields, refs):
        np.testing.assert_allclose(dt.jacobian(f), ref, rtol=0, atol=1e-13)
