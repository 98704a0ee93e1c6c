"""The FFT form of the FDK pre-filter: every transform size and ragged rows against
the FP64 oracle, and rows that are not finite (kept out of the transform their pair
shares).  Tolerance: the operators' 1e-5 relative L2."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _run(sino, ang, geom, filt):
    import torch
    from mexct import ops

    d = torch.from_numpy(np.ascontiguousarray(sino.transpose(2, 1, 0))).cuda()
    return ops.prefilter_dev(d, ang, geom, 700.0, filt).cpu().numpy().transpose(2, 1, 0)


# orders 64, 64, 128, 256, 512, 1024, 2048, 4096; 2049: the direct form
@pytest.mark.parametrize("W,nP", [(5, 7), (32, 3), (33, 5), (127, 4), (256, 3), (385, 3),
                                  (1000, 2), (2048, 2), (2049, 2)])
def test_every_order_matches_oracle(cuda, orc, W, nP):
    rng = np.random.default_rng(W)
    sino = np.asfortranarray(rng.uniform(0, 2, (W, W, nP)).astype(np.float32))
    ang = np.linspace(0, 3.5, nP).astype(np.float32)
    geom, filt = W % 3, ["ramp", "hamming", "none"][W % 2 + (W == 33)]
    got = _run(sino, ang, geom, filt)
    ref = orc.prefilter(sino, geom, ang, filt, 1.0, 1.0, sad=700.0)
    assert rel_l2(got, ref) <= 1e-5


def test_rows_that_are_not_finite_stay_by_themselves(cuda):
    """NaN, infinite or very large values in one row change that row alone, and a row
    of large finite values equals the scaled row."""
    W, nP = 100, 3
    rng = np.random.default_rng(1)
    sino = np.asfortranarray(rng.uniform(0, 2, (W, W, nP)).astype(np.float32))
    ang = np.linspace(0, 3.5, nP).astype(np.float32)
    clean = _run(sino, ang, 2, "ramp")
    dirty = sino.copy(order="F")
    dirty[3, 10, 0] = np.nan
    dirty[99, 13, 1] = np.inf
    dirty[:, 20, 2] *= np.float32(2.0) ** 110
    got = _run(dirty, ang, 2, "ramp")
    assert np.isnan(got[:, 10, 0]).all()
    assert not np.isfinite(got[:, 13, 1]).any()
    scaled = got[:, 20, 2].astype(np.float64) / 2.0 ** 110
    assert rel_l2(scaled, clean[:, 20, 2]) <= 1e-5
    keep = np.ones(sino.shape[1:], bool)
    keep[10, 0] = keep[13, 1] = keep[20, 2] = False
    assert rel_l2(got[:, keep], clean[:, keep]) <= 1e-5
