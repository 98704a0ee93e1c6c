"""OSC-TV on volumes whose rows are not a multiple of four voxels: the TV steps use the
solver's own buffers, so such a volume needs no more memory than its neighbours."""
import numpy as np
import pytest


def test_request_bytes_grow_with_the_width(lib):
    """A request that fits a budget at one width fits it at every smaller one."""
    from mexct import serve

    for kind in (0, 1):
        b = [serve.Server.request_bytes(kind, W, 100, 60, n_sub=10) for W in range(100, 133)]
        assert all(x <= y for x, y in zip(b, b[1:]))


@pytest.mark.gpu
@pytest.mark.parametrize("geom", [0, 2])
@pytest.mark.parametrize("W", [33, 34, 35, 36])
def test_volumes_between_steps_stay_whole(cuda, geom, W):
    """With a TV constant of 0 the 20 steps move the volume between the buffers and add
    nothing, so the solver's iterates are the OSC operator's, bit for bit: eager, captured
    and in one host call."""
    import torch
    from mexct import ops, phantoms, solver

    H, nP, sad = 24, 24, 1000.0
    ang = phantoms.angles_full(nP)
    rng = np.random.default_rng(W)
    pre = np.full((W, H, nP), 1e5, dtype=np.float32, order="F")
    post = np.asfortranarray((pre * np.exp(-rng.uniform(0.5, 2, pre.shape))).astype(np.float32))
    d = [torch.from_numpy(np.ascontiguousarray(a.transpose(2, 1, 0))).cuda() for a in (pre, post)]
    firsts = [1, 2, 3]
    mu = torch.full((H, W, W), 1e-10, device="cuda")
    p, q = d[0].clone(), d[1].clone()
    for k, first in enumerate(firsts):
        if k:
            p.view(-1)[0] = q.view(-1)[0] = 0.0  # the driver zeroes them from iteration 2 on
        ops.osc_iter_dev(mu, p, q, 4, solver.subset_order(4, first), ang, sad, geom)
    want = mu.cpu().numpy().transpose(2, 1, 0)
    kw = dict(n_iter=3, tv_const=0.0, n_sub_init=4, n_sub_final=4, p_val=1.0)
    for graph in (False, True):
        s = solver.OscTvSolver(d[0], d[1], ang, sad, geom)
        s.run(firsts, use_graph=graph, **kw)
        got = s.mu().cpu().numpy().transpose(2, 1, 0)
        s.close()
        assert np.array_equal(got, want)
    host = solver.OSC_TV_recon(pre, post, ang, {"type": ["par3d", "fan3d", "cone3d"][geom],
                                               "SAD": sad}, 3, 0.0, 4, 4, 1.0, firsts)
    assert np.array_equal(host, want)
