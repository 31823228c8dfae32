"""GPU tests of the particle grouping a non-deterministic world does before its substeps: dense
counting per grid node, the radix sort where the grid is huge for its particles.

Tolerances: trajectories that differ only in the order of atomic sums agree to 1e-6 of the largest
coordinate (a few tens of substeps); the reference modes against the f32 oracle to 2e-5.
"""
import numpy as np
import pytest

import ae_mpm as M
import ae_mpm_scenes as S
import oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a.astype(np.float64) - b).max() / np.abs(b).max())


@pytest.mark.parametrize("interval,threads,graph", [(1, 128, 1), (3, 256, 1), (16, 128, 1), (5, 256, 0)])
def test_uneven_scenes_with_empty_slots_match_scenes_alone(ctx, interval, threads, graph):
    # counts below, at and far below the capacity, an empty scene, one-block grids next to large
    # ones: every scene's sorted places must be its own slot range
    pairs = [S.tiny_scene(n, g, mat, seed=0xB0 + n, v=(0.4, -0.3, 0.2)) for n, g, mat in
             ((1, 4, S.water()), (1000, 16, S.jelly()), (2, 8, S.jelly()), (4097, 36, S.snow()), (33, 7, S.water()),
              (6001, 64, S.jelly()))]
    caps = (7, 1000, 300, 5000, 257, 6001)
    scenes = []
    for (sc, _), cap in zip(pairs, caps):
        sc.wall_margin = 1
        sc.max_particles = cap
        scenes.append(sc)
    opts = dict(sort_interval=interval, block_threads=threads, use_graph=graph)
    w = M.World(ctx, scenes, M.exec_opts(**opts))
    empty = 2
    for i, (_, p) in enumerate(pairs):
        if i != empty:
            w.upload(i, p)
    for k in (7, 34):  # odd first run: later periods start on the other parity
        w.step(k)
    w.upload(3, pairs[3][1])  # one scene restarts: the order starts anew for the whole world
    w.step(10)
    assert w.sync(raise_on_error=False) in (M.OK, M.EDOMAIN)
    for i, (sc, p) in enumerate(pairs):
        if i == empty:
            continue
        alone = M.World(ctx, [sc], M.exec_opts(sort_interval=1, use_graph=0))
        alone.upload(0, p)
        alone.step(10 if i == 3 else 51)
        alone.sync(raise_on_error=False)
        a, b = w.download(i, p.n), alone.download(0, p.n)
        assert rel(a.pos, b.pos) <= 1e-6, i
        assert np.array_equal(a.mass, b.mass), i
        alone.close()
    w.close()


def test_huge_grid_with_few_particles_matches_small_grid_order(ctx):
    # 256^3 nodes for 2 000 particles: the radix sort is kept; held to the FP64 oracle
    sc, p = S.tiny_scene(2000, 256, S.snow(), v=(0.5, 0.0, -0.5), box=(0.45, 0.48))
    ref = p.astype(np.float64)
    O.run(sc, ref, 20)
    for interval in (1, 4):
        w = M.World(ctx, [sc], M.exec_opts(sort_interval=interval))
        w.upload(0, p)
        w.step(20)
        w.sync()
        assert rel(w.download(0, p.n).pos, ref.pos) <= 1e-5, interval
        w.close()


@pytest.mark.parametrize("n", [33, 5000, 70001])
def test_off_grid_particles_of_the_reference_modes_match_the_oracle(ctx, n):
    # a tenth of the particles lies beyond the grid's upper faces and shares the dead key with the
    # world's empty slots (the capacity is the power of two above n)
    rng = np.random.default_rng(n)
    g, dx = 24, 0.5
    p = M.Particles.empty(n)
    p.pos[:] = (0.5 + rng.random((n, 3)) * (g - 4)) * dx
    out = rng.random(n) < 0.1
    p.pos[out, rng.integers(0, 3)] += g * dx
    p.vel[:] = rng.normal(0, 0.3, (n, 3))
    p.mass[:] = 0.01
    p.J[:] = 1.0
    cfg = M.Config(grid_dx=dx, grid_size=(g, g, g), substeps=3, gravity=(0, -9.81, 0), damping=0.995)
    grid = M.Grid(g, g, g, dx, (0.0, 0.0, 0.0))
    mats = [M.material(young_modulus=1e4, poisson_ratio=0.25, density=1000.0)]
    idx = np.arange(n, dtype=np.uint64)
    a, b = p.copy(), p.copy()
    ctx.step_parallel_with_grid(a, grid, cfg, mats, [M.NEO_HOOKEAN], 0.016, idx)
    assert O.step_parallel_with_grid(b, grid, cfg, mats, [M.NEO_HOOKEAN], 0.016, idx) == 0
    assert rel(a.pos, b.pos) <= 2e-5
    a, b = p.copy(), p.copy()
    ctx.step_velocity_only_parallel(a, grid, cfg, 0.1, idx)
    assert O.step_velocity_only_parallel(b, grid, cfg, 0.1, idx) == 0
    assert rel(a.pos, b.pos) <= 2e-5


@pytest.mark.parametrize("sizes", [(1, 31, 32, 33), (512, 64, 2), (513, 700, 40), (3000, 5)])
def test_deterministic_sums_over_crowded_cells(ctx, sizes):
    # cells of up to 32 particles, up to the rank limit and above it: the slot order of each cell, and
    # with it every bit, repeats from run to run whatever order the grouping's atomics gave
    rng = np.random.default_rng(sum(sizes))
    g, dx = 16, 1.0 / 16
    x = np.concatenate([(np.array([4.6 + 1.5 * i, 5.6, 6.6]) + 0.8 * rng.random((k, 3))) * dx
                        for i, k in enumerate(sizes)])
    x = x[rng.permutation(len(x))]
    p = S.make_particles(x, (0.3, -0.2, 0.1), 1e-5, 0)
    p.J[:] = 1.0
    sc = M.Scene(n=(g, g, g), dx=dx, dt=1e-4, materials=[S.jelly(E=100.0)], max_particles=p.n + 9)
    ref = p.astype(np.float64)
    O.run(sc, ref, 7)
    runs = []
    for graph in (0, 1, 1):
        w = M.World(ctx, [sc], M.exec_opts(deterministic=1, use_graph=graph))
        w.upload(0, p)
        w.step(7)
        w.sync(raise_on_error=False)
        runs.append(w.download(0, p.n))
        w.close()
    assert rel(runs[0].pos, ref.pos) <= 1e-5
    for r in runs[1:]:
        for f in ("pos", "vel", "F", "J", "C"):
            assert np.array_equal(getattr(r, f), getattr(runs[0], f)), f


@pytest.mark.parametrize("mode", [M.MODE_REFERENCE, M.MODE_VELOCITY_ONLY])
def test_deterministic_reference_modes_with_off_grid_particles_repeat(ctx, mode):
    rng = np.random.default_rng(7)
    g, dx, n = 20, 0.5, 3001
    p = M.Particles.empty(n)
    p.pos[:] = rng.random((n, 3)) * (g + 2) * dx  # some beyond the upper faces
    p.vel[:] = rng.normal(0, 0.3, (n, 3))
    p.mass[:] = 0.01
    p.J[:] = 1.0
    sc = M.Scene(n=(g, g, g), dx=dx, dt=0.01, materials=[M.material(young_modulus=1e4, poisson_ratio=0.25)], mode=mode,
                 gravity=(0, -9.81, 0), max_particles=n + 100)
    out = []
    for det in (1, 1, 0):
        w = M.World(ctx, [sc], M.exec_opts(deterministic=det))
        w.upload(0, p)
        w.step(5)
        w.sync(raise_on_error=False)
        out.append(w.download(0, n))
        w.close()
    for f in ("pos", "vel", "F", "J", "C"):
        assert np.array_equal(getattr(out[0], f), getattr(out[1], f)), f
    assert rel(out[0].pos, out[2].pos) <= 2e-5


@pytest.mark.parametrize("grid", [20, 216])
def test_deterministic_world_takes_particles_far_outside_its_grid(ctx, grid):
    # physics mode clamps a position into the grid in its first G2P; until then a stencil may lie wholly
    # outside: such particles add nothing to the grid, mark no block of it, and come back at its border.
    # Two scenes of 216^3 nodes with these few particles take the radix-sorted form of the same sums.
    rng = np.random.default_rng(grid)
    n, dx = 900, 1.0 / grid
    x = (8.0 + 4.0 * rng.random((n, 3))) * dx
    far = np.arange(0, n, 9)
    x[far, rng.integers(0, 3, far.size)] = np.where(rng.random(far.size) < 0.5, -7.3, grid + 9.4) * dx
    p = S.make_particles(x, (0.2, -0.1, 0.3), 1e-5, 0)
    p.J[:] = 1.0
    sc = M.Scene(n=(grid, grid, grid), dx=dx, dt=1e-4, materials=[S.jelly(E=100.0)], max_particles=n)
    out = []
    for det in (1, 1, 0):
        w = M.World(ctx, [sc, sc], M.exec_opts(deterministic=det))
        w.upload(0, p)
        w.upload(1, p)
        w.step(4)
        assert w.sync(raise_on_error=False) == M.EDOMAIN
        out.append((w.download(0, n), w.download(1, n)))
        w.close()
    for f in ("pos", "vel", "F", "J", "C"):
        assert np.array_equal(getattr(out[0][0], f), getattr(out[1][1], f)), f
    assert rel(out[0][0].pos, out[2][0].pos) <= 1e-6


def crowd(n, g, k, seed):
    # n particles spread over a grid of g nodes per axis, k of them in one cell
    rng = np.random.default_rng(seed)
    dx = 1.0 / g
    x = (4.0 + (g - 8.0) * rng.random((n, 3))) * dx
    x[rng.choice(n, k, replace=False)] = (6.6 + 0.8 * rng.random((k, 3))) * dx
    p = S.make_particles(x, (0.2, -0.1, 0.1), 1e-5, 0)
    p.J[:] = 1.0
    return M.Scene(n=(g, g, g), dx=dx, dt=1e-5, materials=[S.jelly(E=10.0)], max_particles=n), p


@pytest.mark.parametrize("n,k", [(513, 513), (1500, 640), (40000, 5000), (70001, 4097), (70001, 69000)])
def test_deterministic_sums_over_one_crowded_cell_repeat(ctx, n, k):
    # slots of one and of two scenes, sorted in two and in three passes of 8 bits
    sc, p = crowd(n, 24, k, n + k)
    other, q = crowd(900, 16, 700, 3)
    ref = p.astype(np.float64)
    O.run(sc, ref, 3)
    runs = []
    for scenes in ([sc], [sc], [other, sc]):
        w = M.World(ctx, scenes, M.exec_opts(deterministic=1))
        if len(scenes) == 2:
            w.upload(0, q)
        w.upload(len(scenes) - 1, p)
        w.step(3)
        w.sync(raise_on_error=False)
        runs.append(w.download(len(scenes) - 1, n))
        w.close()
    assert rel(runs[0].pos, ref.pos) <= 1e-5
    for r in runs[1:]:
        for f in ("pos", "vel", "F", "J", "C"):
            assert np.array_equal(getattr(r, f), getattr(runs[0], f)), f


@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("mode", [M.MODE_REFERENCE, M.MODE_VELOCITY_ONLY])
@pytest.mark.parametrize("n,share", [(700, 1.0), (5003, 0.5), (40000, 0.9)])
def test_deterministic_reference_modes_with_many_off_grid_particles_repeat(ctx, mode, n, share, threads):
    # most of a scene above the grid's top, where the reference lets it fall back in
    rng = np.random.default_rng(n)
    g, dx = 20, 0.5
    p = M.Particles.empty(n)
    p.pos[:] = (0.5 + (g - 4) * rng.random((n, 3))) * dx
    above = rng.random(n) < share
    p.pos[above, 1] = (g + 0.6 + 0.5 * rng.random(int(above.sum()))) * dx
    p.vel[:] = rng.normal(0, 0.3, (n, 3))
    p.vel[:, 1] -= 20.0
    p.mass[:] = 0.01
    p.J[:] = 1.0
    sc = M.Scene(n=(g, g, g), dx=dx, dt=0.01, materials=[M.material(young_modulus=1e3, poisson_ratio=0.25)], mode=mode,
                 gravity=(0, -9.81, 0), max_particles=n + 100)
    out = []
    for det in (1, 1, 0):
        w = M.World(ctx, [sc, sc], M.exec_opts(deterministic=det, block_threads=threads))
        w.upload(0, p)
        w.upload(1, p)
        w.step(5)
        w.sync(raise_on_error=False)
        out.append((w.download(0, n), w.download(1, n)))
        w.close()
    for f in ("pos", "vel", "F", "J", "C"):
        assert np.array_equal(getattr(out[0][0], f), getattr(out[1][0], f)), f
        assert np.array_equal(getattr(out[0][0], f), getattr(out[0][1], f)), f
    assert rel(out[0][0].pos, out[2][0].pos) <= 2e-5


def test_deterministic_substeps_do_not_stall_on_one_crowded_cell(ctx):
    # 600 particles of 1 M in one cell cost about what 500 cost (walking the scene for them took 40 times
    # as long), and so do 600 particles above the grid in a reference mode
    import torch

    def time_us(sc, p):
        w = M.World(ctx, [sc], M.exec_opts(deterministic=1))
        w.upload(0, p)
        w.step(4)
        st = torch.cuda.ExternalStream(w.stream())
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(st)
        w.step(6)
        b.record(st)
        b.synchronize()
        w.close()
        return a.elapsed_time(b) * 1000.0 / 6

    n = 1000000
    few, many = (time_us(*crowd(n, 96, k, 1)) for k in (500, 600))
    assert many <= 4.0 * few
    sc, p = crowd(n, 96, 1, 1)
    sc.mode, sc.gravity, p.vel[:] = M.MODE_REFERENCE, (0, 0, 0), 0.0
    few = time_us(sc, p)
    p.pos[:600, 1] += 1.0
    assert time_us(sc, p) <= 4.0 * few


def test_stage_times_count_the_grouping_as_the_sort(ctx):
    # every substep groups 1 M particles (scan and placement, some 20 us) or none does: the grid update's
    # time is the same either way
    sc, p = crowd(1000000, 96, 1, 2)
    t = {}
    for interval in (1, 64):
        w = M.World(ctx, [sc], M.exec_opts(sort_interval=interval))
        w.upload(0, p)
        w.step(4)
        t[interval] = w.stage_times(20)
        w.close()
    assert t[1]["sort"] > 5.0
    assert t[1]["grid"] <= 1.3 * t[64]["grid"]


@pytest.mark.parametrize("mode,deterministic,interval", [(M.MODE_PHYSICS, 0, 1), (M.MODE_PHYSICS, 0, 3), (M.MODE_PHYSICS, 0, 8),
                                                         (M.MODE_PHYSICS, 1, 1), (M.MODE_REFERENCE, 0, 4),
                                                         (M.MODE_REFERENCE, 1, 1)])
def test_graphs_carry_the_sort_of_their_period(ctx, mode, deterministic, interval):
    # a run of whole periods consists of graph launches alone
    import torch
    from torch.profiler import ProfilerActivity, profile

    sc, p = crowd(20000, 32, 1, 4)
    sc.mode = mode
    w = M.World(ctx, [sc], M.exec_opts(sort_interval=interval, deterministic=deterministic))
    w.upload(0, p)
    w.step(96)
    w.step(48)  # periods that start on the other parity are captured by now
    w.sync(raise_on_error=False)
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        w.step(48)
        w.sync(raise_on_error=False)
        torch.cuda.synchronize()
    w.close()
    names = [e.name for e in prof.events()]
    if not any("Launch" in n for n in names):
        pytest.skip("the profiler recorded no runtime calls here")
    assert sum("GraphLaunch" in n for n in names) == 48 // (interval if interval % 2 == 0 else 2 * interval)
    assert sum("LaunchKernel" in n for n in names) == 0


@pytest.mark.parametrize("mode", [M.MODE_PHYSICS, M.MODE_REFERENCE])
def test_deterministic_world_on_a_huge_grid_repeats_and_matches(ctx, mode):
    # 8.5 M nodes and more for a few thousand particles: the radix-sorted sums, one thread per cell,
    # with crowded cells and (reference mode) particles off the grid
    sc, p = crowd(4000, 216, 700, 11)
    sc.mode, sc.max_particles = mode, p.n + 5
    if mode == M.MODE_REFERENCE:
        p.pos[::50, 1] += 1.0
    runs = []
    for det in (1, 1, 0):
        w = M.World(ctx, [sc, sc], M.exec_opts(deterministic=det))
        w.upload(0, p)
        w.upload(1, p)
        w.step(6)
        w.sync(raise_on_error=False)
        runs.append((w.download(0, p.n), w.download(1, p.n)))
        w.close()
    for f in ("pos", "vel", "F", "J", "C"):
        assert np.array_equal(getattr(runs[0][0], f), getattr(runs[1][0], f)), f
        assert np.array_equal(getattr(runs[0][0], f), getattr(runs[0][1], f)), f
    assert rel(runs[0][0].pos, runs[2][0].pos) <= 1e-6
