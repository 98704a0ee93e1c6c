"""The rows FP without clusters, the form that full-size calls take (one, two and four views
per CTA, tiles and chunks that end early, both sweep axes in one CTA), and with them: steep
fans with lists too long and boxes too narrow, voxels that are not finite, FP16 / BF16
storage, the OSC epilogue, columns of a decoupled detector.  The cases assert the form that
they run on.  The oracle gets some of the views.  Tolerances: 1e-5 relative L2 in FP32 (every
operator's), 1e-3 with FP16 and 1e-2 with BF16 storage, 1e-4 for an OSC iteration."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _vol(W, H, seed=0):
    return np.asfortranarray(np.random.default_rng(seed + W).uniform(0, 1, (W, W, H))
                             .astype(np.float32))


def _dev(vol, dtype="float32"):
    import torch

    return torch.from_numpy(np.ascontiguousarray(vol.transpose(2, 1, 0))).to(
        getattr(torch, dtype)).cuda()


def _host(t):
    return t.float().cpu().numpy().transpose(2, 1, 0)


def _deg(start, step, n):
    return np.deg2rad(start + step * np.arange(n, dtype=np.float64)).astype(np.float32)


def _rows(form, W, H, sad, ang, geom, nsub=0):
    """The call runs on the rows kernel with (views per CTA, CTAs per cluster) = form."""
    from mexct import tune

    assert tune.fp_plan(W, H, sad, ang, geom, nsub) == (True,) + form


# W around the 32-column tile, H around the 128-row chunk; spacings that put 1, 2 or 4 views
# in a CTA, view counts that leave the last CTA short, angles on both sides of 45 and 135
# degrees and across them (views that sweep different axes in one CTA)
CASES = [(33, 130, 0.5, 630, 4), (64, 127, 0.25, 1001, 4), (65, 129, 0.5, 423, 4),
         (65, 60, 0.5, 250, 2), (40, 126, 35.0, 403, 1), (97, 70, 20.0, 205, 1),
         (31, 257, 0.3, 1203, 4)]


@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("W,H,spacing,nP,views", CASES)
def test_tiles_chunks_and_views(cuda, orc, geom, W, H, spacing, nP, views):
    from mexct import _lib, ops

    sad, vol = 3.0 * W, _vol(W, H)
    ang = _deg(40.0, spacing, nP)
    _rows((views, 1), W, H, sad, ang, geom)
    got = _host(ops.fp_dev(_dev(vol), sad, ang, geom, variant=_lib.FP_EXPLICIT))
    # some of the first, middle and last views, and those around the changes of axis
    deg = np.rad2deg(ang.astype(np.float64)) % 180
    pick = set(range(3)) | set(range(nP - 5, nP)) | {nP // 2}
    for turn in (45.0, 135.0):
        pick |= set(np.argsort(np.abs(deg - turn))[:6].tolist())
    pick = np.array(sorted(pick))
    ref = orc.fp(vol, sad, ang[pick], len(pick), geom)
    for i, k in enumerate(pick):
        assert rel_l2(got[:, :, k], ref[:, :, i]) <= 1e-5, k


@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("dtype,tol", [("float16", 1e-3), ("bfloat16", 1e-2)])
@pytest.mark.parametrize("spacing,nP,views", [(0.5, 423, 4), (25.0, 300, 1)])
def test_16_bit_storage(cuda, orc, geom, dtype, tol, spacing, nP, views):
    import torch
    from mexct import _lib, ops

    W, H, sad, ang = 65, 131, 200.0, _deg(20.0, spacing, nP)
    _rows((views, 1), W, H, sad, ang, geom)
    d = _dev(_vol(W, H), dtype)
    for out in (d.dtype, torch.float32):
        got = _host(ops.fp_dev(d, sad, ang, geom, out_dtype=out, variant=_lib.FP_EXPLICIT))
        pick = np.arange(0, nP, 37)
        ref = orc.fp(np.asfortranarray(_host(d)), sad, ang[pick], len(pick), geom)
        # FP32 output of a 16-bit volume: the FP32 bound
        assert rel_l2(got[:, :, pick], ref) <= (tol if out == d.dtype else 1e-5)


@pytest.mark.parametrize("sad,nP,spacing,views", [(45.0, 240, 1.5, 1), (70.0, 240, 1.5, 1),
                                                  (300.0, 400, 0.4, 2)])
def test_steep_fans(cuda, orc, sad, nP, spacing, views):
    """Rays up to ~75 degrees from the sweep axis: lists too long for a plane, boxes that
    do not hold the tile."""
    from mexct import _lib, ops

    W, H, ang = 80, 70, _deg(3.0, spacing, nP)
    _rows((views, 1), W, H, sad, ang, 1)
    vol = _vol(W, H)
    got = _host(ops.fp_dev(_dev(vol), sad, ang, 1, variant=_lib.FP_EXPLICIT))
    pick = np.arange(0, nP, 11)
    ref = orc.fp(vol, sad, ang[pick], len(pick), 1)
    for i, k in enumerate(pick):
        assert rel_l2(got[:, :, k], ref[:, :, i]) <= 1e-5, k


@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("spacing,nP,views", [(0.5, 423, 4), (25.0, 300, 1)])
def test_a_voxel_that_is_not_finite_reaches_its_own_rays_only(cuda, geom, spacing, nP, views):
    from mexct import _lib, ops

    W, H, sad, ang = 65, 129, 500.0, _deg(0.0, spacing, nP)
    _rows((views, 1), W, H, sad, ang, geom)
    vol = _vol(W, H)
    clean = _host(ops.fp_dev(_dev(vol), sad, ang, geom, variant=_lib.FP_EXPLICIT))
    x, y, z = 40, 22, 128
    vol[x, y, z] = np.inf
    got = _host(ops.fp_dev(_dev(vol), sad, ang, geom, variant=_lib.FP_EXPLICIT))
    px, py = x - (W - 1) / 2, y - (W - 1) / 2
    for k, b in enumerate(ang.astype(np.float64)):
        s, t = px * np.cos(b) + py * np.sin(b), py * np.cos(b) - px * np.sin(b)
        u = t * (sad / (sad - s) if geom else 1.0) + (W - 1) / 2
        far = np.abs(np.arange(W) - u) > 3.0
        assert rel_l2(got[far, z, k], clean[far, z, k]) <= 1e-6
        assert not np.isfinite(got[int(round(u)), z, k])
    rest = np.arange(H) != z
    assert np.array_equal(got[:, rest], clean[:, rest])


@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("nP,nsub,views", [(1440, 2, 4), (500, 2, 2), (180, 2, 1)])
def test_osc_residuals(cuda, orc, geom, nP, nsub, views):
    """An OSC iteration whose subsets run without clusters (EPI 1), oracle in full."""
    import mexct

    W, H, sad = {4: (33, 130, 400.0), 2: (65, 100, 400.0), 1: (65, 129, 400.0)}[views]
    ang = np.linspace(0, 2 * np.pi, nP, endpoint=False).astype(np.float32)
    _rows((views, 1), W, H, sad, ang, geom, nsub)
    rng = np.random.default_rng(views)
    mu = np.asfortranarray(rng.uniform(0, 0.02, (W, W, H)).astype(np.float32))
    pre = np.full((W, H, nP), 1e5, np.float32, order="F")
    post = np.asfortranarray((pre * np.exp(-rng.uniform(0.3, 1, pre.shape))).astype(np.float32))
    picks = np.arange(nsub, dtype=np.int32)
    ref = orc.osc_iter(mu, pre, post, nsub, picks, ang, sad, geom)
    mexct.CUDAmex_oscIter(mu, pre, post, nsub, picks, ang, sad, geom)
    assert rel_l2(mu, ref) <= 1e-4


# few views: clusters of eight, of four with four buffers (4 x views x tiles <= SMs) and two
@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("W,H,nP,split", [(64, 130, 9, 8), (100, 201, 4, 8), (65, 130, 12, 4),
                                          (65, 129, 40, 4)])
def test_clusters(cuda, orc, geom, W, H, nP, split):
    from mexct import _lib, ops

    sad, vol = 2.0 * W, _vol(W, H)
    ang = np.concatenate([_deg(41.0, 2.0, nP // 2), _deg(130.0, 2.5, nP - nP // 2)])
    _rows((1, split), W, H, sad, ang, geom)
    got = _host(ops.fp_dev(_dev(vol), sad, ang, geom, variant=_lib.FP_EXPLICIT))
    assert rel_l2(got, orc.fp(vol, sad, ang, nP, geom)) <= 1e-5
    vol[W // 2, W // 3, H - 1] = np.nan
    bad = _host(ops.fp_dev(_dev(vol), sad, ang, geom, variant=_lib.FP_EXPLICIT))
    assert np.array_equal(bad[:, :-1], got[:, :-1]) and np.isnan(bad[:, -1]).any()
    far = np.isfinite(bad[:, -1])
    assert far.sum() > 0.8 * far.size and rel_l2(bad[:, -1][far], got[:, -1][far]) <= 1e-6


@pytest.mark.parametrize("sad", [45.0, 70.0])
def test_steep_fans_in_clusters(cuda, orc, sad):
    from mexct import _lib, ops

    W, H, ang = 80, 60, _deg(0.0, 16.0, 23)
    _rows((1, 4), W, H, sad, ang, 1)
    vol = _vol(W, H)
    got = _host(ops.fp_dev(_dev(vol), sad, ang, 1, variant=_lib.FP_EXPLICIT))
    assert rel_l2(got, orc.fp(vol, sad, ang, len(ang), 1)) <= 1e-5


@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("nP", [11, 301])
@pytest.mark.parametrize("Wd,du", [(75, 0.8), (90, 1.3), (20, 1.0), (33, 2.5)])
def test_decoupled_columns(cuda, orc, geom, nP, Wd, du):
    """Columns of their own: rays that miss the volume, tiles wider than the staged box; as
    many detector rows as slices, enough of them for the rows kernel."""
    from mexct import ops

    W, H, vol = 48, 130, _vol(48, 130)
    ang = _deg(10.0, 29.0, nP)
    got = _host(ops.fp_det_dev(_dev(vol), 300.0, ang, geom, Wd, H, du, 1.0, 1))
    pick = np.arange(0, nP, max(1, nP // 11))
    ref = orc.fp_det(vol, 300.0, ang[pick], geom, Wd, H, du, 1.0, 1)
    assert rel_l2(got[:, :, pick], ref) <= 1e-5
