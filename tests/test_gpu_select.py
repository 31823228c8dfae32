"""GPU tests of the near cap's selection (lod_classify): where the keys' digits, the candidates kept in
shared memory and the ties at the cap change sides.  Index lists: no tolerance.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.mark.parametrize("n,cap,spread", [
    (2, 1, "wide"), (33, 32, "wide"), (1024, 1023, "wide"), (1025, 1, "one"), (3000, 1500, "one"),
    (40960, 20000, "wide"), (40961, 20001, "wide"), (90000, 89999, "bits11"), (5000, 2500, "bits11"),
    (5000, 2500, "bits12"), (50000, 7, "exponents"), (4096, 4096, "wide"), (4096, 5000, "wide"),
])
def test_near_cap_keeps_the_closest_and_ties_by_index(ctx, n, cap, spread):
    # wide: distances over the whole near range.  one: all distances equal.  bits11 / bits12: squared
    # distances that differ in their lowest 11 / 12 bits only, each many times.  exponents: 2^-60 .. 2^10.
    rng = np.random.default_rng(n + cap)
    pos = np.zeros((n, 3), f32)
    if spread == "wide":
        pos[:] = rng.uniform(-25, 25, (n, 3))
    elif spread == "one":
        pos[:, 1] = 3.0
    elif spread == "exponents":
        pos[:, 2] = np.exp2(rng.uniform(-30, 5, n))
    else:
        # x^2 of x in [1, 1 + 2^-12) covers 2^11 steps of 2^-23 (bits12: 2^12 steps)
        pos[:, 0] = 1.0 + rng.integers(0, 1 << (10 if spread == "bits11" else 11), n) * 2.0 ** -23
    player = np.zeros(3, f32)
    rn, rm, rf = O.lod_classify(pos, None, player, 50.0, 200.0, cap)
    gn, gm, gf = ctx.lod_classify(pos, None, player, 50.0, 200.0, cap)
    d = pos - player
    d2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
    keep = np.sort(np.argsort(d2, kind="stable")[:cap])
    assert rf.size == gf.size == 0
    assert np.array_equal(gn, keep)
    assert np.array_equal(gm, np.setdiff1d(np.arange(n), keep))
    assert np.array_equal(np.sort(d2[gn]), np.sort(d2[rn])) and gm.size == rm.size


@pytest.mark.parametrize("n,near,cap", [(3000, 100, 1000), (3000, 100, 100), (3000, 2500, 100), (5000, 4000, 0),
                                        (5000, 4000, 5000), (100000, 60000, 59999)])
def test_lists_in_device_memory_are_written_up_to_their_counts(ctx, n, near, cap):
    import ctypes as C

    import torch

    rng = np.random.default_rng(n + cap)
    pos = rng.uniform(200, 300, (n, 3)).astype(f32)
    pos[rng.choice(n, near, replace=False)] = rng.uniform(-20, 20, (near, 3))
    player = np.zeros(3, f32)
    want = O.lod_classify(pos, None, player, 50.0, 400.0, cap)
    dpos = torch.from_numpy(pos).cuda()
    lists = [torch.full((n,), -7, dtype=torch.int64, device="cuda") for _ in range(3)]
    counts = [C.c_uint64() for _ in range(3)]
    torch.cuda.synchronize()
    ctx.check(ctx.lib.ae_mpm_lod_classify(ctx.h, dpos.data_ptr(), None, n, player.ctypes.data, 50.0, 400.0, cap,
                                          lists[0].data_ptr(), C.byref(counts[0]), lists[1].data_ptr(), C.byref(counts[1]),
                                          lists[2].data_ptr(), C.byref(counts[2])))
    for k, (got, c) in enumerate(zip(lists, counts)):
        a = got.cpu().numpy()
        ref = np.asarray(want[k]).astype(np.int64)
        assert c.value == ref.size
        assert np.array_equal(np.sort(a[:c.value]), np.sort(ref)), k  # the oracle's culled tail has its own order
        assert (a[c.value:] == -7).all(), k
