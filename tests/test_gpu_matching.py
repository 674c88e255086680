"""The matching solver (volume_matching_3d) on the device against the
reference's own results (tests/golden/matching.npz, made from
src/VolumeMatching3D.c by tests/golden/make_golden.py).

Both compute in FP32; the reference sums the cost sequentially in float and
the device in FP64, so the step-control decisions can differ in the last
bits of a comparison: fields agree to 2e-3 (typically to float rounding) and
the final masked residuals to 1e-3."""
from __future__ import annotations

import os

import numpy as np
import pytest

import disptools_b200 as dt
from tests.helpers import ball_problem, masked_max

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def cases():
    d = np.load(os.path.join(HERE, "golden", "matching.npz"))
    count = len({name.split("_")[0] for name in d.files})
    return [tuple(d[f"m{k}_{n}"] for n in ("Jt", "mask", "field0", "spacing", "it_max", "out"))
            for k in range(count)]


def test_matching_matches_reference(cases, oracle):
    for Jt, m, f0, sp, it, ref in cases:
        out, st = dt.solve(Jt, m, f0, spacing=tuple(sp), algorithm="matching", it_max=int(it))
        assert st["iterations"] == int(it)
        assert np.max(np.abs(out - ref)) <= 2e-3
        r_ref = masked_max(oracle.jacobian(ref, tuple(sp)), Jt, m)
        r_out = masked_max(oracle.jacobian(out, tuple(sp)), Jt, m)
        assert abs(r_out - r_ref) <= 1e-3, (r_out, r_ref)


def test_matching_entry_points_agree(cases):
    """The extension, the reference-named C function and the Python API give
    the same field."""
    from disptools_b200 import _disptools
    from disptools_b200 import _native as N
    Jt, m, f0, sp, it, _ = cases[1]
    a, _ = dt.solve(Jt, m, f0, spacing=tuple(sp), algorithm="matching", it_max=int(it))
    b = np.ascontiguousarray(f0.copy())
    args = [9.99e-4, 0.2, 0.1, 0.4, 1.2, 0.5, 0.1, 1e-3, 10.0, 1e-6, 1e-9]
    _disptools.displacement(tuple(sp), Jt, m, *args, False, int(it), b, "matching", -1)
    c = np.ascontiguousarray(f0.copy())
    nz, ny, nx = Jt.shape
    N.lib.volume_matching_3d(nx, ny, nz, *map(float, sp), Jt.ctypes.data, m.ctypes.data, *args, False,
                             int(it), c.ctypes.data)
    assert not N.lib.disptools_has_error()
    np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(a, c)


def test_matching_cost_decreases_and_stops():
    Jt, m = ball_problem(24, 12, 6, 0.9)
    _, s0 = dt.solve(Jt, m, algorithm="matching", it_max=0)
    out, s1 = dt.solve(Jt, m, algorithm="matching", it_max=25)
    assert s0["iterations"] == 0 and s1["iterations"] == 25
    assert s1["error"] < s0["error"]
    assert np.isfinite(out).all()
    # a loose epsilon stops the solver before it_max
    _, s2 = dt.solve(Jt, m, algorithm="matching", it_max=500, epsilon=0.05)
    assert s2["iterations"] < 500 and s2["max_error"] <= 0.05


def test_matching_device_entry_equals_host(cases):
    """dtb_volume_matching_device (through torch_ops.solve on float64
    tensors, on a side stream) gives the host entry's field bit for bit;
    float32 tensors are refused."""
    import torch

    from disptools_b200 import torch_ops
    Jt, m, f0, sp, it, _ = cases[3]
    a, sa = dt.solve(Jt, m, f0, spacing=tuple(sp), algorithm="matching", it_max=int(it))
    Jd, md = torch.from_numpy(Jt).cuda(), torch.from_numpy(m).cuda()
    fd = torch.from_numpy(f0.copy()).cuda()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        st = torch_ops.solve(Jd, md, fd, spacing=tuple(sp), algorithm="matching", it_max=int(it))
    torch.cuda.current_stream().wait_stream(side)
    np.testing.assert_array_equal(fd.cpu().numpy(), a)
    assert (st["iterations"], st["reason"]) == (sa["iterations"], sa["reason"])
    with pytest.raises(ValueError):
        torch_ops.solve(Jd.float(), md, fd.float(), spacing=tuple(sp), algorithm="matching", it_max=1)


def test_matching_profile_counts_kernels():
    """With profiling on, every gradient and cost launch of the matching
    solver is timed."""
    Jt, m = ball_problem(20, 10, 5, 1.1)
    dt.set_profiling(True)
    try:
        _, st = dt.solve(Jt, m, algorithm="matching", it_max=5)
        prof = dt.kernel_profile()
    finally:
        dt.set_profiling(False)
    assert st["iterations"] == 5
    g, c = prof["match_gradient"], prof["match_cost"]
    assert g[0] >= 5 and c[0] >= g[0] + 1
    assert g[1] > 0.0 and c[1] > 0.0


def _optimiser64(J, params):
    """The optimiser of src/VolumeMatching3D.c:408-557 on a zero field, unit
    spacing, cost and gradient in float64 by torch's autograd."""
    import torch
    nz, ny, nx = J.shape
    grid = torch.meshgrid(*[torch.arange(1, n + 1, dtype=torch.float64) for n in (nz, ny, nx)], indexing="ij")
    pos = torch.stack([grid[1], grid[2], grid[0]])  # y, x, z
    V = torch.as_tensor(J)[:-1, :-1, :-1]
    eps, zeta = params["delta"], params["zeta"]

    def cost(p):
        edge = [p[:, :, 1:] - p[:, :, :-1], p[:, :, :, 1:] - p[:, :, :, :-1], p[:, 1:] - p[:, :-1]]  # along y, x, z
        s, barrier = 0.0, 0.0
        for k in (0, 1):
            for x in (0, 1):
                for y in (0, 1):
                    m = [edge[0][:, k:nz - 1 + k, :, x:nx - 1 + x], edge[1][:, k:nz - 1 + k, y:ny - 1 + y],
                         edge[2][:, :, y:ny - 1 + y, x:nx - 1 + x]]
                    Jc = torch.linalg.det(torch.stack(m, dim=-1).movedim(0, -2))
                    s = s + Jc
                    barrier = barrier + torch.where(Jc < eps, zeta * (Jc - eps) ** 2, torch.zeros_like(Jc))
        volume = torch.where(V > 0, (s - 8 * V) ** 2, torch.zeros_like(s))
        return 0.5 * (volume + barrier).sum(), float(((s - 8 * V).abs() / 8).max().detach())

    def trial(g, alpha):
        h, worst = cost(pos - alpha * g)
        return float(h), worst

    alpha, it, phases = 1.0, 0, set()
    H, worst = trial(torch.zeros_like(pos), 0.0)
    while it < params["it_max"] and alpha > 1e-9 and worst > params["epsilon"]:
        q = pos.clone().requires_grad_()
        (g,) = torch.autograd.grad(cost(q)[0], q)
        mark = H
        h, worst = trial(g, alpha)
        step = alpha
        if h < mark and it == 0:
            phases.add("double")
            while h < mark:
                mark, alpha = h, alpha * 2
                h, worst = trial(g, alpha)
            step = alpha = alpha * 0.5
            h = mark
        elif h < mark:
            phases.add("grow")
            alpha = float(np.float32(alpha) * 1.05)
        else:
            while h > mark and alpha > 1e-9:
                phases.add("halve")
                alpha *= 0.5
                h, worst = trial(g, alpha)
            step = alpha
        if alpha > 1e-9:
            pos, H, it = pos - step * g, h, it + 1
    return pos, it, phases


# zeta 1e-3 with a floor of 2 and no volume term (J <= 0): the first step
# of 1 lowers the cost, so it is doubled; the other start halves it.
@pytest.mark.parametrize("target, delta, zeta, wanted", [(0.0, 2.0, 1e-3, "double"), (1.2, 1e-3, 10.0, "halve")])
def test_device_step_control_against_float64(target, delta, zeta, wanted):
    """The doubling, growing and halving branches of the device's step control
    against a float64 restatement, for a few iterations (the solver computes
    in float32)."""
    J = np.full((4, 5, 6), target)
    J[2, 2, 3] += 0.3 * (target > 0)
    params = dict(delta=delta, zeta=zeta, it_max=3, epsilon=9.99e-4)
    pos, it, phases = _optimiser64(J, params)
    assert wanted in phases
    out, st = dt.solve(J, np.ones(J.shape, bool), algorithm="matching", **params)
    assert st["iterations"] == it
    z, y, x = np.meshgrid(*[np.arange(1, n + 1) for n in J.shape], indexing="ij")
    ref = np.stack([pos[1].numpy() - x, pos[0].numpy() - y, pos[2].numpy() - z])
    assert np.max(np.abs(out - ref)) <= 1e-4


@pytest.mark.parametrize("it_max", [2 ** 56, 2 ** 62, 2 ** 63 - 1])
def test_matching_takes_any_iteration_limit(it_max):
    """A limit far beyond reach ("no limit") is the same as one just out of
    reach: the bound on queued steps does not wrap."""
    Jt, m = ball_problem(16, 8, 4, 1.1)
    kw = dict(algorithm="matching", epsilon=0.02)
    want, sw = dt.solve(Jt, m, it_max=100000, **kw)
    assert 16 < sw["iterations"] < 100000
    got, sg = dt.solve(Jt, m, it_max=it_max, **kw)
    assert sg["iterations"] == sw["iterations"]
    np.testing.assert_array_equal(got, want)


def test_matching_of_a_long_column():
    """2 x 2 x 4.3 million voxels, more gradient runs than a grid has z blocks:
    away from the one place that moves nothing does, so the first planes are
    those of the short column (only the cost's summation order differs)."""
    import torch

    from disptools_b200 import torch_ops
    results = []
    for nz in (400, 4_300_000):
        J = torch.ones((nz, 2, 2), dtype=torch.float64, device="cuda")
        J[40:60] = 1.05
        field = torch.zeros((3, nz, 2, 2), dtype=torch.float64, device="cuda")
        st = torch_ops.solve(J, torch.ones(J.shape, dtype=torch.bool, device="cuda"), field, algorithm="matching",
                             it_max=4)
        results.append((field, st["iterations"]))
    (short, it_short), (long, it_long) = results
    assert it_long == it_short > 0
    assert float(short.abs().max()) > 0.0
    torch.testing.assert_close(long[:, :300], short[:, :300], rtol=0, atol=1e-5)
    assert not long[:, 300:].any()


def test_matching_from_many_threads():
    """More solves at once than pinned states are kept: each the field of the
    solve alone."""
    from concurrent.futures import ThreadPoolExecutor
    problems = [ball_problem(n, n / 2, n / 4, 1.1) for n in (10, 12, 14, 16)]
    kw = dict(algorithm="matching", it_max=12)
    alone = [dt.solve(J, m, **kw)[0] for J, m in problems]
    with ThreadPoolExecutor(16) as pool:
        for got, want in zip(pool.map(lambda p: dt.solve(*p, **kw)[0], problems * 8), alone * 8):
            np.testing.assert_array_equal(got, want)
