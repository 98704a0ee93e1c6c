"""Parallel / fan FP over the z-fastest layout: tile and chunk edges, one / two / four
views per CTA, long weight lists, volumes that are not finite.  Tolerances: 1e-5 relative
L2 against the FP64 oracle in FP32 (every operator's), 1e-3 with FP16 storage."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _dev(vol):
    import torch

    return torch.from_numpy(np.ascontiguousarray(vol.transpose(2, 1, 0))).cuda()


def _host(t):
    return t.float().cpu().numpy().transpose(2, 1, 0)


# W around the 32-column tile, H around the 128-row chunk (rows 1 .. H of H + 2); the
# angles' spacing puts 1, 2 or 4 views in a CTA and crosses 45 and 135 degrees
@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("W,H,spacing", [(31, 1, 1.0), (33, 126, 0.2), (32, 127, 3.0),
                                         (65, 130, 2.0), (40, 7, 40.0), (1, 3, 10.0)])
def test_edges_match_oracle(cuda, orc, geom, W, H, spacing):
    from mexct import ops

    rng = np.random.default_rng(W + H)
    vol = np.asfortranarray(rng.uniform(0, 1, (W, W, H)).astype(np.float32))
    ang = np.deg2rad(np.concatenate([41 + spacing * np.arange(5), 131 + spacing * np.arange(4)]))
    ang = ang.astype(np.float32)
    got = _host(ops.fp_dev(_dev(vol), 300.0, ang, geom))
    assert rel_l2(got, orc.fp(vol, 300.0, ang, len(ang), geom)) <= 1e-5


@pytest.mark.parametrize("sad", [45.0, 70.0, 150.0])
def test_steep_fans(cuda, orc, sad):
    """Rays up to ~75 degrees from the sweep axis: long lists, boxes that do not hold the
    tile, and (the shortest) rays that are taken sample by sample."""
    from mexct import ops

    W, H = 80, 20
    rng = np.random.default_rng(4)
    vol = np.asfortranarray(rng.uniform(0, 1, (W, W, H)).astype(np.float32))
    ang = np.linspace(0, 2 * np.pi, 23).astype(np.float32)
    got = _host(ops.fp_dev(_dev(vol), sad, ang, 1))
    assert rel_l2(got, orc.fp(vol, sad, ang, len(ang), 1)) <= 1e-5


@pytest.mark.parametrize("geom", [0, 1])
def test_half_storage(cuda, orc, geom):
    import torch
    from mexct import ops

    W, H = 45, 131
    rng = np.random.default_rng(5)
    vol = np.asfortranarray(rng.uniform(0, 1, (W, W, H)).astype(np.float16).astype(np.float32))
    ang = np.linspace(0, np.pi, 31).astype(np.float32)
    got = _host(ops.fp_dev(_dev(vol).half(), 500.0, ang, geom, out_dtype=torch.float16))
    assert rel_l2(got, orc.fp(vol, 500.0, ang, len(ang), geom)) <= 1e-3


@pytest.mark.parametrize("geom", [0, 1])
def test_a_voxel_that_is_not_finite_reaches_its_own_rays_only(cuda, geom):
    """One NaN voxel: the rays more than two voxels away from it are what they are
    without it, and the rays through it are NaN."""
    from mexct import ops

    W, H = 64, 9
    rng = np.random.default_rng(6)
    vol = np.asfortranarray(rng.uniform(0, 1, (W, W, H)).astype(np.float32))
    ang = np.deg2rad(np.arange(0, 180, 7.0)).astype(np.float32)
    clean = _host(ops.fp_dev(_dev(vol), 500.0, ang, geom))
    x, y, z = 40, 22, 4
    vol[x, y, z] = np.nan
    got = _host(ops.fp_dev(_dev(vol), 500.0, ang, geom))
    px, py = x - (W - 1) / 2, y - (W - 1) / 2
    for k, b in enumerate(ang.astype(np.float64)):
        s, t = px * np.cos(b) + py * np.sin(b), py * np.cos(b) - px * np.sin(b)
        u = t * (500.0 / (500.0 - s) if geom else 1.0) + (W - 1) / 2
        far = np.abs(np.arange(W) - u) > 3.0
        assert np.array_equal(got[far, z, k] == got[far, z, k], np.ones(far.sum(), bool))
        assert rel_l2(got[far, z, k], clean[far, z, k]) <= 1e-6
        assert np.isnan(got[int(round(u)), z, k])
    rest = np.arange(H) != z
    assert np.array_equal(got[:, rest], clean[:, rest])


@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("Wd,du", [(75, 0.8), (90, 1.3), (20, 1.0), (33, 2.5)])
def test_decoupled_columns(cuda, orc, geom, Wd, du):
    """Detector rows that are the volume's slices, columns of their own: rays that miss
    the volume, and tiles wider than the staged box."""
    from mexct import ops

    W, H = 48, 21
    rng = np.random.default_rng(Wd)
    vol = np.asfortranarray(rng.uniform(0, 1, (W, W, H)).astype(np.float32))
    ang = np.deg2rad(10 + 29.0 * np.arange(11)).astype(np.float32)
    got = _host(ops.fp_det_dev(_dev(vol), 300.0, ang, geom, Wd, H, du, 1.0, 1))
    assert rel_l2(got, orc.fp_det(vol, 300.0, ang, geom, Wd, H, du, 1.0, 1)) <= 1e-5
