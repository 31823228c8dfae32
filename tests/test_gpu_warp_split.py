"""GPU tests at the sizes where a world's kernels change how many particles a warp takes, and of the
warp vote that maps yielding snow back in place or queues it.

Tolerances: the deterministic world sums the same terms in another order: positions within 1e-6 of the
largest coordinate over a few tens of substeps, 2e-5 in the reference modes.  Snow against the FP64
oracle over three substeps: positions 1e-5; deformation gradients and J 2e-5, a few tens of roundings
of entries near 1 through an SVD and its reassembly per substep.
"""
import numpy as np
import pytest
import torch

import ae_mpm as M
import ae_mpm_scenes as S
import oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a.astype(np.float64) - b).max() / np.abs(b).max())


@pytest.mark.parametrize("per_sm,over", [(80, 0), (80, 1), (320, 0), (320, 1)])
def test_fused_kernel_at_the_sizes_where_its_split_changes(ctx, per_sm, over):
    n = torch.cuda.get_device_properties(0).multi_processor_count * per_sm + over
    sc, p = S.tiny_scene(n, 32, S.jelly(), v=(0.4, -0.3, 0.2))
    out = []
    for det in (0, 1):
        w = M.World(ctx, [sc], M.exec_opts(deterministic=det))
        w.upload(0, p)
        w.step(18)
        w.sync()
        out.append(w.download(0, n))
        w.close()
    assert rel(out[0].pos, out[1].pos) <= 1e-6


@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("mode", [M.MODE_REFERENCE, M.MODE_VELOCITY_ONLY])
def test_reference_scatter_at_the_size_where_its_split_changes(ctx, mode, over):
    n = torch.cuda.get_device_properties(0).multi_processor_count * 128 + over
    rng = np.random.default_rng(n)
    g, dx = 40, 0.5
    p = M.Particles.empty(n)
    p.pos[:] = (1 + rng.random((n, 3)) * (g - 5)) * dx
    p.vel[:] = rng.normal(0, 0.3, (n, 3))
    p.mass[:] = 0.01
    p.J[:] = 1.0
    sc = M.Scene(n=(g, g, g), dx=dx, dt=0.002, materials=[M.material(young_modulus=1e3, poisson_ratio=0.25)], mode=mode,
                 gravity=(0, -9.81, 0), max_particles=n)
    out = []
    for det in (0, 1):
        w = M.World(ctx, [sc], M.exec_opts(deterministic=det))
        w.upload(0, p)
        w.step(3)
        w.sync(raise_on_error=False)
        out.append(w.download(0, n))
        w.close()
    assert rel(out[0].pos, out[1].pos) <= 2e-5


@pytest.mark.parametrize("share", [0.02, 0.25, 0.5, 1.0])
def test_snow_yielding_in_part_of_a_warp_matches_the_oracle(ctx, share):
    # a quarter of 32 lanes is the vote's limit: warps below, at and above it
    sc, p = S.tiny_scene(4001, 16, S.snow(), v=(0.2, -0.1, 0.1))
    rng = np.random.default_rng(int(share * 100))
    p.F[:] = np.eye(3, dtype=np.float32).reshape(p.F.shape[1:])
    hit = rng.random(p.n) < share
    p.F[hit] = np.diag([1.05, 1.0, 0.94]).astype(np.float32).reshape(p.F.shape[1:])
    ref = p.astype(np.float64)
    O.run(sc, ref, 3)
    w = M.World(ctx, [sc], M.exec_opts())
    w.upload(0, p)
    w.step(3)
    w.sync()
    got = w.download(0, p.n)
    w.close()
    assert rel(got.pos, ref.pos) <= 1e-5
    assert rel(got.F, ref.F) <= 2e-5
    assert rel(got.J, ref.J) <= 2e-5
