"""The fused TV steps (one gradient per step): row lengths that are and are not a multiple
of four, x tiles (128, 256, 512 and wider), slices per CTA, step counts, in place, and a
buffer that is not 16-byte aligned.  Tolerance: 1e-5 relative L2 against the FP64 oracle
for up to three steps (every FP32 operator's); more steps amplify rounding, so 20 steps
are compared at 1e-4 on a volume with noise everywhere."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _vol(Nx, Ny, Nz):
    rng = np.random.default_rng(Nx + Ny + Nz)
    return np.asfortranarray(rng.uniform(0, 1, (Nx, Ny, Nz)).astype(np.float32))


@pytest.mark.parametrize("shape,steps", [((4, 4, 4), 1), ((5, 3, 3), 2), ((128, 15, 33), 2),
                                         ((127, 8, 5), 3), ((129, 9, 32), 2), ((256, 22, 4), 1),
                                         ((259, 7, 31), 3), ((512, 8, 3), 2), ((513, 16, 9), 2),
                                         ((1021, 10, 5), 3), ((1, 9, 9), 2), ((60, 50, 40), 20),
                                         ((61, 50, 40), 20)])
def test_steps_match_oracle(cuda, orc, shape, steps):
    import mexct

    vol = _vol(*shape)
    got = mexct.CUDAmex_TVmin_3D(vol, 0.05, steps)
    ref = orc.tvmin3d(vol, 0.05, steps)
    both = np.isfinite(ref)  # a volume without interior voxels has norm 0: scale * 0 is NaN
    assert np.array_equal(both, np.isfinite(got))
    assert rel_l2(got[both], ref[both]) <= (1e-5 if steps <= 3 else 1e-4)


@pytest.mark.parametrize("steps", [1, 2, 5])
@pytest.mark.parametrize("Nx", [64, 66])
def test_in_place_and_unaligned_equal_out_of_place(cuda, steps, Nx):
    import torch
    from mexct import ops

    vol = torch.from_numpy(np.ascontiguousarray(_vol(Nx, 20, 37).transpose(2, 1, 0))).cuda()
    ref = ops.tvmin3d_dev(vol, 0.05, steps)
    own = vol.clone()
    ops.tvmin3d_dev(own, 0.05, steps, out=own)
    flat = torch.empty(vol.numel() + 1, device="cuda")
    off = flat[1:].view(vol.shape)
    off.copy_(vol)
    out = torch.empty(vol.numel() + 1, device="cuda")[1:].view(vol.shape)
    ops.tvmin3d_dev(off, 0.05, steps, out=out)
    assert torch.equal(own, ref) and torch.equal(out, ref)


def test_captured_call_matches(cuda):
    """A captured call allocates nothing: it takes the pair of sweeps, and replays."""
    import torch
    import mexct

    vol = torch.from_numpy(np.random.default_rng(8).uniform(0, 1, (20, 33, 44)).astype(np.float32)).cuda()
    out = torch.empty_like(vol)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    mexct.ops.tvmin3d_dev(vol, 0.05, 3, out=out, stream=st)
    st.synchronize()
    want = out.clone()
    out.zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        mexct.ops.tvmin3d_dev(vol, 0.05, 3, out=out, stream=st)
    g.replay()
    torch.cuda.synchronize()
    assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) <= 1e-5
