"""GPU test of the CK-MPM gather kernel's record pipeline: groups of 32 records, several per warp, at
remainders and at record arrays that start on no 16-byte boundary.  The deterministic mode runs it
every step and equals the oracle (with the device's correctly rounded logarithm) bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

import ae_mpm as M
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 4097, 227400 + 13])
def test_gather_pipeline_is_bit_exact(ctx, n, offset):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    h, side = 1.0, 64
    pos = 8.0 + 40.0 * rng.random((n, 3))
    p0 = M.ck_particles(pos, 0.5, 0.125, velocity=rng.normal(0, 1.0, (n, 3)))
    p0[:, 6:15] = rng.normal(0, 0.05, (n, 9))
    p0[:, 15:24] += rng.normal(0, 0.01, (n, 9)).astype(np.float32)
    cfg = M.ck_config(dt=5e-3, grid_n=side, grid_h=h, bounds_min=(0, 0, 0), bounds_max=(side,) * 3)
    want = p0.copy()
    O.ck_step(want, cfg, 2, correctly_rounded_ln=True)
    buf = torch.zeros(p0.size + 4, dtype=torch.float32, device="cuda")
    view = buf[offset:offset + p0.size]
    view.copy_(torch.from_numpy(p0.ravel()))
    ctx.check(ctx.lib.ae_mpm_ck_step_deterministic(ctx.h, view.data_ptr(), n, C.byref(cfg), 2))
    got = view.cpu().numpy().reshape(p0.shape)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert float(buf[:offset].abs().sum()) == 0.0 and float(buf[offset + p0.size:].abs().sum()) == 0.0
