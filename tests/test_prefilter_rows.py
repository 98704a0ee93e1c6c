"""Two detector rows share one complex transform in the pre-filter's FFT form: a row's
result must not depend on how large its partner is.  Every row of a pair is held by itself
to the operators' 1e-5 relative L2 against the FP64 oracle, whatever the other row's scale,
and a row of zeros stays exactly zero."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _run(sino, ang, geom, filt):
    import torch
    from mexct import ops

    d = torch.from_numpy(np.ascontiguousarray(sino.transpose(2, 1, 0))).cuda()
    return ops.prefilter_dev(d, ang, geom, 700.0, filt).cpu().numpy().transpose(2, 1, 0)


# orders 64 (two warps' worth of transforms per warp) to 4096, even and odd row counts
@pytest.mark.parametrize("W,filt", [(5, "ramp"), (32, "hann"), (101, "hamming"), (384, "hamming"),
                                    (1025, "ramp")])
@pytest.mark.parametrize("scale", [1e2, 1e4, 1e8, 2.0 ** 90, 1e-30, 0.0])
def test_a_row_keeps_its_accuracy_beside_a_larger_one(cuda, orc, W, filt, scale):
    geom, views = W % 3, (1, 2)  # the first and last view's dbeta is zero here
    rng = np.random.default_rng(W)
    sino = rng.uniform(0.5, 2, (W, W, 4)).astype(np.float32)
    f = np.float32(scale)
    sino[:, 0::2, 1] *= f  # the pair's upper row in view 1, its lower row in view 2
    sino[:, 1::2, 2] *= f
    sino = np.asfortranarray(sino)
    ang = np.linspace(0, 3.5, 4).astype(np.float32)
    got = _run(sino, ang, geom, filt)
    ref = orc.prefilter(sino, geom, ang, filt, 1.0, 1.0, sad=700.0)
    for k in views:
        for v in range(W):
            if scale == 0.0 and v % 2 == k - 1:
                assert not got[:, v, k].any()
            else:
                assert ref[:, v, k].any()
                assert rel_l2(got[:, v, k], ref[:, v, k]) <= 1e-5, (v, k)
