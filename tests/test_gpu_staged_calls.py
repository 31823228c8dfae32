"""GPU tests of the drop-in calls at the list lengths where the selected particles start to travel in
pieces, for contiguous, sparse and whole selections, against the f32 oracle.

Tolerances: 2e-5 of the largest value (order of the atomic sums over a few substeps); particles that
were not selected, and the arrays that a velocity-only call does not own, keep every bit.
"""
import numpy as np
import pytest

import ae_mpm as M
import oracle as O

pytestmark = pytest.mark.gpu
FIELDS = ("pos", "vel", "F", "J", "C", "mass", "mat")
MOTION, FULL = (64 << 10) // 28, (2 << 20) // 106


def rel(a, b):
    return float(np.abs(a.astype(np.float64) - b).max() / np.abs(b).max())


def buffer(capacity, seed):
    rng = np.random.default_rng(seed)
    g, dx = 24, 0.5
    p = M.Particles.empty(capacity)
    p.pos[:] = (0.5 + rng.random((capacity, 3)) * (g - 4)) * dx
    p.vel[:] = rng.normal(0, 0.3, (capacity, 3))
    p.mass[:] = 0.01
    p.F[:] = np.eye(3, dtype=np.float32).reshape(9)
    p.J[:] = 1.0
    p.C[:] = rng.normal(0, 0.01, (capacity, 9))
    cfg = M.Config(grid_dx=dx, grid_size=(g, g, g), substeps=2, gravity=(0, -9.81, 0), damping=0.995)
    return p, M.Grid(g, g, g, dx, (0.0, 0.0, 0.0)), cfg


@pytest.mark.parametrize("pick", ["sparse", "middle", "all"])
@pytest.mark.parametrize("full,n", [(0, MOTION), (0, MOTION + 1), (0, 41003), (1, FULL), (1, FULL + 1), (1, 40001)])
def test_staged_lists_match_the_oracle_and_leave_the_rest(ctx, full, n, pick):
    capacity = n if pick == "all" else 2 * n + 77
    p, grid, cfg = buffer(capacity, n)
    rng = np.random.default_rng(n + 1)
    if pick == "sparse":
        idx = np.sort(rng.choice(capacity, n, replace=False)).astype(np.uint64)
    else:
        first = 0 if pick == "all" else 31
        idx = np.arange(first, first + n, dtype=np.uint64)
    mats = [M.material(young_modulus=1e3, poisson_ratio=0.25, density=1000.0)]
    a, b = p.copy(), p.copy()
    if full:
        ctx.step_parallel_with_grid(a, grid, cfg, mats, [M.NEO_HOOKEAN], 0.004, idx)
        assert O.step_parallel_with_grid(b, grid, cfg, mats, [M.NEO_HOOKEAN], 0.004, idx) == 0
    else:
        ctx.step_velocity_only_parallel(a, grid, cfg, 0.05, idx)
        assert O.step_velocity_only_parallel(b, grid, cfg, 0.05, idx) == 0
    sel = idx.astype(np.int64)
    rest = np.setdiff1d(np.arange(capacity), sel)
    assert rel(a.pos, b.pos) <= 2e-5
    assert rel(a.vel, b.vel) <= 2e-5
    if full:
        assert rel(a.F, b.F) <= 2e-5 and rel(a.J, b.J) <= 2e-5
    for f in FIELDS:
        assert np.array_equal(getattr(a, f)[rest], getattr(p, f)[rest]), f
        if f in ("mass", "mat") or (not full and f not in ("pos", "vel")):
            assert np.array_equal(getattr(a, f), getattr(p, f)), f


@pytest.mark.parametrize("pick", ["sparse", "all"])
@pytest.mark.parametrize("n", [FULL + 1, 40001, 150001])
def test_staged_reference_calls_bring_the_affine_matrix_back(ctx, n, pick):
    # C is one of the two largest arrays on the way back, cut over several pieces.  It is a velocity
    # gradient: sums of some 30 f32 terms at 4e-6 of the node velocity, times 6 / dx, against a largest
    # entry of about one node velocity over dx, so 1e-4 of it; a row out of place differs by its size
    capacity = n if pick == "all" else 2 * n + 77
    p, grid, cfg = buffer(capacity, n)
    rng = np.random.default_rng(n + 2)
    idx = (np.arange(n) if pick == "all" else np.sort(rng.choice(capacity, n, replace=False))).astype(np.uint64)
    mats = [M.material(young_modulus=1e3, poisson_ratio=0.25, density=1000.0)]
    a, b = p.copy(), p.copy()
    ctx.step_parallel_with_grid(a, grid, cfg, mats, [M.NEO_HOOKEAN], 0.004, idx)
    assert O.step_parallel_with_grid(b, grid, cfg, mats, [M.NEO_HOOKEAN], 0.004, idx) == 0
    sel = idx.astype(np.int64)
    assert rel(a.C, b.C) <= 1e-4
    assert (np.abs(b.C[sel] - p.C[sel]).max(1) > 0).all() and (np.abs(a.C[sel] - p.C[sel]).max(1) > 0).all()
