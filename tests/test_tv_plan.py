"""Which form the FP32 TV descent takes: one fused sweep per step, or a norm and an update
sweep where the columns that the tiles waste make that pair faster (measured on 152 SMs).
The two forms are held to the oracle and to each other (the operators' 1e-5 relative L2)."""
import numpy as np
import pytest

from conftest import rel_l2

# (Nz, Ny, Nx), steps: faster by a tenth or more in that form
FUSED = [((256, 256, 256), 20), ((256, 256, 256), 1), ((64, 64, 64), 20), ((384, 384, 384), 20),
         ((512, 512, 512), 20), ((16, 256, 256), 1), ((64, 384, 384), 1), ((20, 600, 600), 20),
         ((300, 601, 601), 1), ((50, 1001, 1001), 20), ((100, 240, 248), 20)]
PAIR = [((300, 600, 600), 20), ((300, 600, 600), 1), ((200, 360, 372), 20), ((100, 360, 372), 1),
        ((300, 495, 496), 20), ((200, 750, 744), 20), ((640, 640, 640), 1), ((448, 448, 448), 1),
        ((20, 2000, 2000), 1)]


@pytest.mark.parametrize("shape,steps", FUSED + PAIR)
def test_the_faster_form(lib, shape, steps):
    from mexct import tune

    assert tune.tv_plan(*shape[::-1], n_steps=steps, sms=152) == ((shape, steps) in FUSED)


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [1, 2, 3])
def test_both_forms_agree(cuda, orc, steps):
    """248 x 240 x 330 columns fill the pair's tiles; a volume that is not 16-byte aligned
    takes the fused form."""
    import torch
    from mexct import ops, tune

    shape = (330, 240, 248)
    assert not tune.tv_plan(*shape[::-1], n_steps=steps)
    rng = np.random.default_rng(steps)
    vol = rng.uniform(0, 1, shape).astype(np.float32)
    pair = ops.tvmin3d_dev(torch.from_numpy(vol).cuda(), 0.05, steps).cpu().numpy()
    off = torch.empty(vol.size + 1, device="cuda")[1:].view(shape)
    off.copy_(torch.from_numpy(vol))
    fused = ops.tvmin3d_dev(off, 0.05, steps).cpu().numpy()
    ref = orc.tvmin3d(np.asfortranarray(vol.transpose(2, 1, 0)), 0.05, steps).transpose(2, 1, 0)
    assert rel_l2(pair, ref) <= 1e-5
    assert rel_l2(fused, ref) <= 1e-5
    assert rel_l2(fused, pair) <= 1e-5
