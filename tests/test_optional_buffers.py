"""Buffers that a context keeps only for speed (general3D BP pairs, TV gradients): a call
that cannot have them takes the form without, another operator's allocation that fails
gets their memory back, and large ones do not outlive their call.  Failures are injected
on the host (mexct_fail_allocs)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

S, Z, W, H, NP = 64, 40, 64, 48, 100  # 307200 rays: more than the pair form asks for


@pytest.fixture
def fail():
    from mexct import _lib

    yield lambda n: _lib.call("mexct_fail_allocs", n)
    _lib.call("mexct_fail_allocs", 0)


def _bp_inputs():
    import torch

    rng = np.random.default_rng(2)
    pts = np.zeros((W, H, 6), np.float32, order="F")
    pts[..., 0], pts[..., 3] = 150.0, -150.0
    pts[..., 1:3] = rng.uniform(-20, 20, (W, H, 2))
    pts[..., 4:6] = rng.uniform(-20, 20, (W, H, 2))
    sino = np.asfortranarray(rng.uniform(0, 1, (W, H, NP)).astype(np.float32))
    ang = np.linspace(0, np.pi, NP).astype(np.float32)
    return (pts, sino, ang, torch.from_numpy(pts.ravel(order="F")).cuda().view(6, H, W),
            torch.from_numpy(sino.ravel(order="F")).cuda().view(NP, H, W))


def _ctx():
    """A context of its own: nothing is kept from other tests."""
    import ctypes

    from mexct import _lib

    c = ctypes.c_void_p()
    _lib.call("mexct_ctx_create", 0, ctypes.byref(c))
    return c


def _g3d(c, ds, ang, dp, out):
    import torch
    from mexct import _lib, ops

    _lib.call("mexct_g3d_bp_dev", c, ops._dptr(ds), W, H, NP, ops._ptr(ang), ops._dptr(dp), 0, S, Z,
              ops._dptr(out), ops._stream(None))
    torch.cuda.synchronize()
    return out.cpu().numpy().transpose(2, 1, 0)


def _tv(c, vol, out, steps=2):
    import torch
    from mexct import _lib, ops

    nz, ny, nx = vol.shape
    _lib.call("mexct_tvmin3d_dev", c, ops._dptr(vol), nx, ny, nz, 0.05, steps, ops._dptr(out),
              ops._stream(None))
    torch.cuda.synchronize()


def _fp(c):
    """A cone FP in a context; (result, oracle's arguments)."""
    import torch
    from mexct import _lib, ops

    vol = torch.from_numpy(np.random.default_rng(5).uniform(0, 1, (32, 24, 24)).astype(np.float32))
    vol, a = vol.cuda(), np.linspace(0, np.pi, 9).astype(np.float32)
    sino = torch.empty((9, 32, 24), device="cuda")
    _lib.call("mexct_fp_dev", c, ops._dptr(vol), 24, 32, 500.0, ops._ptr(a), 9, 2, ops._dptr(sino),
              ops._stream(None))
    torch.cuda.synchronize()
    return (sino.cpu().numpy().transpose(2, 1, 0),
            (vol.cpu().numpy().transpose(2, 1, 0), 500.0, a, 9, 2))


def _flush(fail):
    """Every context gives its optional buffers back to an allocation that fails."""
    from mexct import _lib

    c = _ctx()
    fail(1)
    try:
        _fp(c)
    except _lib.MexctError:  # there were none
        pass
    fail(0)
    _lib.call("mexct_ctx_destroy", c)


def test_a_call_without_them_gives_the_same_result(cuda, orc, fail):
    import torch
    from mexct import _lib

    pts, sino, ang, dp, ds = _bp_inputs()
    ref = orc.g3d_bp(sino, ang, pts, S, Z)
    vol = np.random.default_rng(3).uniform(0, 1, (20, 33, 41)).astype(np.float32)
    tv_ref = orc.tvmin3d(vol.transpose(2, 1, 0), 0.05, 2).transpose(2, 1, 0)
    dvol = torch.from_numpy(vol).cuda()
    for refused in (False, True):
        c, out = _ctx(), torch.empty((Z, S, S), device="cuda")
        fail(int(refused))  # the pair buffers are the call's only allocation
        assert rel_l2(_g3d(c, ds, ang, dp, out), ref) <= 1e-5
        _tv(c, dvol[:1].contiguous(), torch.empty_like(dvol[:1]))  # scalars and partial sums
        _flush(fail)
        tv = torch.empty_like(dvol)
        _tv(c, dvol, tv)
        assert rel_l2(tv.cpu().numpy(), tv_ref) <= 1e-5
        _flush(fail)
        fail(int(refused))  # everything but the gradients is there
        tv.zero_()
        _tv(c, dvol, tv)
        fail(0)
        assert rel_l2(tv.cpu().numpy(), tv_ref) <= 1e-5
        _lib.call("mexct_ctx_destroy", c)


def test_another_allocation_gets_their_memory(cuda, orc, fail):
    """An allocation that fails once succeeds after some context's optional buffers went;
    with nothing to give back it is the out-of-memory error that it was."""
    import torch
    from mexct import _lib

    _, _, ang, dp, ds = _bp_inputs()
    other = _ctx()
    for kept in (False, True):
        c = _ctx()
        _flush(fail)
        if kept:
            _g3d(other, ds, ang, dp, torch.empty((Z, S, S), device="cuda"))
        fail(1)
        if kept:
            got, args = _fp(c)
            assert rel_l2(got, orc.fp(*args)) <= 1e-5
        else:
            with pytest.raises(_lib.MexctError) as ei:
                _fp(c)
            assert ei.value.status == 3  # MEXCT_ERR_OOM
        fail(0)
        _lib.call("mexct_ctx_destroy", c)
    _lib.call("mexct_ctx_destroy", other)


def test_large_buffers_last_for_one_call(cuda):
    """The gradients and second volume of 560 x 1001 x 1001 voxels are 6.7 GB, more than a
    context keeps: after the call only the one volume that every form needs is gone."""
    import torch
    from mexct import _lib, tune

    c = _ctx()
    vol = torch.rand((560, 1001, 1001), device="cuda")
    out = torch.empty_like(vol)
    _tv(c, vol[:1].contiguous(), torch.empty_like(vol[:1]), 1)
    before = torch.cuda.mem_get_info()[0]
    assert tune.tv_plan(1001, 1001, 560, n_steps=10)
    _tv(c, vol, out, 10)
    after = torch.cuda.mem_get_info()[0]
    assert before - after <= 1.1 * 560 * 1001 * 1004 * 4
    _lib.call("mexct_ctx_destroy", c)
