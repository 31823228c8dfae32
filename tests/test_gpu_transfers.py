"""GPU tests of the particle transfers: a world reads and writes views in its device's memory in
place, and views in host memory through a staging area; both give the same bytes.
"""
import ctypes as C

import numpy as np
import pytest

import ae_mpm as M
import ae_mpm_scenes as S

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "F", "J", "C", "mass", "mat")


def device_view(p, offset):
    """Device copies of p's arrays, each starting `offset` elements into an allocation."""
    import torch

    keep = []
    for f in FIELDS:
        a = getattr(p, f).ravel()
        a = a.view(np.int16) if f == "mat" else a
        t = torch.zeros(a.size + offset, dtype=getattr(torch, a.dtype.name), device="cuda")
        t[offset:] = torch.from_numpy(a.copy()).cuda()
        keep.append(t)
    torch.cuda.synchronize()
    return keep, M.ParticlesView(*(t.data_ptr() + offset * t.element_size() for t in keep))


def host_of(keep, offset, like):
    out = like.copy()
    for f, t in zip(FIELDS, keep):
        a = t[offset:].cpu().numpy()
        getattr(out, f)[...] = (a.view(np.uint16) if f == "mat" else a).reshape(getattr(out, f).shape)
    return out


def scene(n, seed, dtype=np.float32):
    sc, p = S.tiny_scene(n, 24, S.jelly(), seed=seed, v=(0.6, -0.4, 0.3))
    rng = np.random.default_rng(seed)
    p.F += rng.normal(0, 1e-3, p.F.shape).astype(np.float32)
    p.C[:] = rng.normal(0, 1.0, p.C.shape)
    perm = rng.permutation(n)  # an order that the sort changes
    return sc, p.subset(perm).astype(dtype)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n,offset", [(1, 0), (31, 1), (33, 0), (257, 3), (5000, 1)])
def test_device_views_in_place_equal_host_views(ctx, n, offset, precision):
    sc, p = scene(n, 0x51 + n, np.float32 if precision == 32 else np.float64)
    opts = M.exec_opts(precision=precision, deterministic=1)
    suffix = "_f64" if precision == 64 else ""
    results = []
    for device in (False, True):
        w = M.World(ctx, [sc], opts)
        if device:
            keep, v = device_view(p, offset)
            ctx.check(getattr(ctx.lib, "ae_mpm_world_upload" + suffix)(
                w.h, 0, C.cast(C.pointer(v), ctx.lib.ae_mpm_world_upload.argtypes[2]) if not suffix else
                C.cast(C.pointer(v), ctx.lib.ae_mpm_world_upload_f64.argtypes[2]), n))
        else:
            w.upload(0, p)
        w.step(6)
        if device:
            out, ov = device_view(p, offset)
            fn = getattr(ctx.lib, "ae_mpm_world_download" + suffix)
            ctx.check(fn(w.h, 0, C.cast(C.pointer(ov), fn.argtypes[2])))
            results.append(host_of(out, offset, p))
            assert all(float(t[:offset].abs().sum()) == 0.0 for t in out)  # nothing before the view
        else:
            results.append(w.download(0, n))
        w.close()
    for f in FIELDS:
        assert np.array_equal(getattr(results[0], f), getattr(results[1], f)), f


def test_many_scene_transfers_mix_device_and_host_views(ctx):
    # device, host and repeated views in one call; scenes out of order and one left out
    pairs = [scene(n, 0x70 + n) for n in (100, 33, 2049, 7, 640)]
    scenes = [sc for sc, _ in pairs]
    ref = M.World(ctx, scenes, M.exec_opts(deterministic=1))
    for i in (0, 1, 2, 4):
        ref.upload(i, pairs[i][1])
    ref.step(5)
    w = M.World(ctx, scenes, M.exec_opts(deterministic=1))
    order = [4, 0, 2, 1, 0]  # scene 0 twice: the last view counts
    dummy = pairs[0][1].copy()
    dummy.pos += np.float32(0.01)
    kept, views = [], (M.ParticlesView * 5)()
    for k, s in enumerate(order):
        src = dummy if k == 1 else pairs[s][1]
        if k % 2 == 0:
            keep, views[k] = device_view(src, 1)
            kept.append(keep)
        else:
            views[k] = src.view()
    ids = np.array(order, np.uint32)
    counts = np.array([pairs[s][1].n for s in order], np.uint64)
    ctx.check(ctx.lib.ae_mpm_world_upload_many(w.h, 5, ids.ctypes.data, C.addressof(views), counts.ctypes.data))
    w.step(5)
    outs, oviews = [], (M.ParticlesView * 5)()
    for k, s in enumerate(order):
        like = pairs[s][1].copy()
        if k % 2 == 0:
            keep, oviews[k] = device_view(like, 1)
            outs.append(("device", keep, like))
        else:
            outs.append(("host", like, like))
            oviews[k] = like.view()
    ctx.check(ctx.lib.ae_mpm_world_download_many(w.h, 5, ids.ctypes.data, C.addressof(oviews)))
    for (kind, a, like), s in zip(outs, order):
        got = host_of(a, 1, like) if kind == "device" else a
        want = ref.download(s, pairs[s][1].n)
        for f in FIELDS:
            assert np.array_equal(getattr(got, f), getattr(want, f)), (s, f)
    ref.close()
    w.close()


def test_a_reported_cuda_error_does_not_fail_the_next_call(ctx):
    # a world that no device can hold is refused; what runs after it starts clean
    sc, p = scene(500, 0x62)
    huge, _ = scene(1, 0x63)
    huge.max_particles = (1 << 31) - 1
    w = M.World(ctx, [sc], M.exec_opts(deterministic=1))
    with pytest.raises(M.MpmError):
        M.World(ctx, [huge])
    w.upload(0, p)
    w.step(2)
    assert w.sync(raise_on_error=False) == M.OK
    w.close()


@pytest.mark.parametrize("short", FIELDS)
@pytest.mark.parametrize("way", ["up", "down"])
def test_device_view_with_a_short_array_is_refused(ctx, way, short):
    # the array's allocation holds half of what the call would read or write: refused, and the context
    # and the world stay usable
    import torch

    torch.zeros(1, device="cuda")
    rt = C.CDLL("libcudart.so.12")
    sc, p = scene(5000, 0x61)
    w = M.World(ctx, [sc], M.exec_opts(deterministic=1))
    w.upload(0, p)
    before = w.download(0, p.n)
    ptrs = []
    for f in FIELDS:
        q = C.c_void_p()
        size = getattr(p, f).nbytes // (2 if f == short else 1)
        assert rt.cudaMalloc(C.byref(q), C.c_size_t(size)) == 0
        assert rt.cudaMemset(q, 0, C.c_size_t(size)) == 0
        ptrs.append(q)
    v = M.ParticlesView(*(q.value for q in ptrs))
    call = ctx.lib.ae_mpm_world_upload if way == "up" else ctx.lib.ae_mpm_world_download
    args = (w.h, 0, C.byref(v)) + ((p.n,) if way == "up" else ())
    assert call(*args) != M.OK
    w.upload(0, p)
    after = w.download(0, p.n)
    for f in FIELDS:
        assert np.array_equal(getattr(after, f), getattr(before, f)), f
    for q in ptrs:
        assert rt.cudaFree(q) == 0
    w.close()


def test_download_into_shared_device_arrays_keeps_the_copy_order(ctx):
    # a caller that wants neither J nor C points both at one buffer, or every scene at one view: the
    # array and the scene that come last are left there whole
    import torch

    pairs = [scene(n, 0x90 + n) for n in (5000, 4097)]
    w = M.World(ctx, [sc for sc, _ in pairs], M.exec_opts(deterministic=1))
    for i, (_, p) in enumerate(pairs):
        w.upload(i, p)
    w.step(3)
    want = [w.download(i, p.n) for i, (_, p) in enumerate(pairs)]
    n = pairs[0][1].n
    keep, v = device_view(pairs[0][1], 0)
    v.jacobian = v.c  # C is copied after J
    extra = torch.zeros(10 * n, dtype=torch.float32, device="cuda")
    v.strain = extra.data_ptr()
    v.mass = extra.data_ptr() + 4 * (9 * n - 12)  # the mass is copied after F: over its last 12 values
    torch.cuda.synchronize()
    ctx.check(ctx.lib.ae_mpm_world_download(w.h, 0, C.byref(v)))
    got = host_of(keep, 0, pairs[0][1])
    assert np.array_equal(got.C, want[0].C) and np.array_equal(got.pos, want[0].pos)
    f = extra.cpu().numpy()
    assert np.array_equal(f[9 * n - 12:10 * n - 12], want[0].mass)
    assert np.array_equal(f[:9 * n - 12], want[0].F.ravel()[:9 * n - 12])
    keep, v = device_view(pairs[0][1], 0)
    views = (M.ParticlesView * 2)(v, v)
    ids = np.array([0, 1], np.uint32)
    ctx.check(ctx.lib.ae_mpm_world_download_many(w.h, 2, ids.ctypes.data, C.addressof(views)))
    got, m = host_of(keep, 0, pairs[0][1]), pairs[1][1].n
    for f in FIELDS:
        assert np.array_equal(getattr(got, f)[:m], getattr(want[1], f)), f
        assert np.array_equal(getattr(got, f)[m:], getattr(want[0], f)[m:]), f
    w.close()


def test_batch_groups_into_one_device_view_keep_the_scene_order(ctx):
    pairs = [scene(n, 0xA0 + n) for n in (3000, 2900, 2800, 2700)]
    parts = [p for _, p in pairs]
    want = [p.copy() for p in parts]
    b = M.Batch(ctx, [sc for sc, _ in pairs], M.exec_opts(deterministic=1), groups=4)
    b.run(parts, 3, out=want)
    keep, v = device_view(parts[0], 0)
    ins, outs = (M.ParticlesView * 4)(*[p.view() for p in parts]), (M.ParticlesView * 4)(v, v, v, v)
    counts = np.array([p.n for p in parts], np.uint64)
    ctx.check(ctx.lib.ae_mpm_batch_run(b.h, C.addressof(ins), counts.ctypes.data, C.addressof(outs), 3))
    got = host_of(keep, 0, parts[0])
    for s in (0, 1, 2, 3):  # scene s shows where the later, shorter ones end
        lo, hi = (parts[s + 1].n if s < 3 else 0), parts[s].n
        for f in FIELDS:
            assert np.array_equal(getattr(got, f)[lo:hi], getattr(want[s], f)[lo:hi]), (s, f)
    b.close()
