"""general3D BP through the pair buffers against the oracle: volumes around the fold's
32 x 32 tile and 16-slice range, rays along x, y, z and diagonals, rays exactly on slices
(kU = kL), and call sizes on both sides of the rule that picks the form.  Tolerance: the
operators' 1e-5 relative L2 in FP32."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


# pairs from S S Z / 16 + 262144 rays: the last two sizes keep the direct form
@pytest.mark.parametrize("S,Z,W,H,nP", [(31, 15, 33, 20, 403), (33, 17, 40, 16, 420), (64, 16, 64, 30, 150),
                                        (5, 1, 90, 73, 40), (65, 49, 40, 20, 6), (40, 90, 9, 5, 3)])
def test_matches_oracle(cuda, orc, S, Z, W, H, nP):
    import mexct

    rng = np.random.default_rng(S + Z)
    half = max(S, Z)
    pts = np.zeros((W, H, 6), dtype=np.float32, order="F")
    pts[..., :3] = rng.uniform(-half, half, (W, H, 3))
    pts[..., 3:] = rng.uniform(-half, half, (W, H, 3))
    z = np.round(rng.uniform(-Z / 2, Z / 2, (W, H))) + (0.5 if Z % 2 else 0.0)  # on a slice
    pts[::3, :, 2] = pts[::3, :, 5] = z[::3]
    pts[1::7, :, 3:5] = pts[1::7, :, 0:2]  # along z
    sino = np.asfortranarray(rng.uniform(-1, 2, (W, H, nP)).astype(np.float32))
    ang = np.linspace(0, 2 * np.pi, nP).astype(np.float32)
    got = mexct.CUDAmex_general3D_BP(sino, ang, pts, S, Z)
    assert rel_l2(got, orc.g3d_bp(sino, ang, pts, S, Z)) <= 1e-5


def test_two_streams(cuda, orc):
    """Calls queued on two streams share the buffers of one context."""
    import torch
    import mexct

    S, Z, W, H, nP = 48, 33, 48, 40, 140
    rng = np.random.default_rng(3)
    pts = np.asfortranarray(rng.uniform(-30, 30, (W, H, 6)).astype(np.float32))
    ang = np.linspace(0, np.pi, nP).astype(np.float32)
    sinos = [np.asfortranarray(rng.uniform(0, 1, (W, H, nP)).astype(np.float32)) for _ in range(4)]
    dp = torch.from_numpy(pts.ravel(order="F")).cuda().view(6, H, W)
    ds = [torch.from_numpy(s.ravel(order="F")).cuda().view(nP, H, W) for s in sinos]
    torch.cuda.synchronize()
    st = [torch.cuda.Stream() for _ in range(2)]
    outs = []
    for i, s in enumerate(ds):
        with torch.cuda.stream(st[i % 2]):
            outs.append(mexct.ops.g3d_bp_dev(s, ang, dp, S, Z, stream=st[i % 2]))
    torch.cuda.synchronize()
    for o, s in zip(outs, sinos):
        want = orc.g3d_bp(s, ang, pts, S, Z)
        assert rel_l2(o.cpu().numpy().transpose(2, 1, 0), want) <= 1e-5
