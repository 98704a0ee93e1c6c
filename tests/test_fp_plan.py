"""Which kernel a parallel / fan FP runs on: the slab kernel for volumes of few slices
(the rows kernel works on 128 slices whatever there are), the rows kernel above.  The
crossovers are those measured on 152 SMs; both kernels' results around them are held to
the oracle (1e-5 relative L2 in FP32, 1e-3 in FP16, 1e-2 in BF16) and, for rays that stay
in a slice, to each other (2e-6: two FP32 sums of the same samples in another order)."""
import numpy as np
import pytest

from conftest import rel_l2


def _ang(n):
    return np.linspace(0, 2 * np.pi, n, endpoint=False).astype(np.float32)


# (W, views, subsets): the most slices for which the slab kernel was faster by more than a
# tenth, and the fewest for which the rows kernel was
@pytest.mark.parametrize("W,nP,nsub,slab,rows", [
    (512, 720, 0, 24, 48), (512, 90, 0, 32, 64), (256, 360, 0, 32, 48), (128, 180, 0, 32, 64),
    (64, 360, 0, 32, 64), (200, 30, 0, 40, 64), (256, 360, 6, 40, 64), (512, 90, 3, 40, 64),
    (64, 60, 0, 4, 64), (256, 60, 10, 1, 32)])
@pytest.mark.parametrize("geom", [0, 1])
def test_thin_volumes_keep_the_slab_kernel(lib, geom, W, nP, nsub, slab, rows):
    from mexct import tune

    for H in {1, slab // 2 or 1, slab}:
        assert not tune.fp_plan(W, H, 1000.0, _ang(nP), geom, nsub, 152)[0], H
    for H in (rows, 2 * rows, 1000):
        assert tune.fp_plan(W, H, 1000.0, _ang(nP), geom, nsub, 152)[0], H


def test_small_problems_and_cone_keep_the_slab_kernel(lib):
    from mexct import tune

    for W, H, nP in ((16, 16, 16), (24, 24, 20), (32, 32, 30), (64, 1, 90), (128, 4, 180)):
        assert not tune.fp_plan(W, H, 1000.0, _ang(nP), 0, 0, 152)[0]
    assert not tune.fp_plan(512, 512, 1000.0, _ang(720), 2, 0, 152)[0]
    # few-view OSC subsets fill idle SMs with clusters at any height
    assert tune.fp_plan(64, 1, 1000.0, _ang(40), 0, 8, 152) == (True, 1, 8)


def _vol(W, H, dtype="float32"):
    import torch

    t = torch.from_numpy(np.random.default_rng(W + H).uniform(0, 1, (H, W, W)).astype(np.float32))
    return t.to(getattr(torch, dtype)).cuda()


def _host(t):
    return t.float().cpu().numpy().transpose(2, 1, 0)


def _both_sides(W, H, nP, sad, geom):
    """(H0, H) with the slab kernel at H0 and the rows kernel at H."""
    from mexct import tune

    thin = max(h for h in range(1, H + 1) if not tune.fp_plan(W, h, sad, _ang(nP), geom)[0])
    assert thin < H and tune.fp_plan(W, H, sad, _ang(nP), geom)[0]
    return thin


@pytest.mark.gpu
@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("dtype,tol", [("float32", 1e-5), ("float16", 1e-3), ("bfloat16", 1e-2)])
def test_fp_on_both_sides_of_the_rule(cuda, orc, geom, dtype, tol):
    import torch
    from mexct import _lib, ops

    W, nP, sad = 70, 150, 300.0
    H0 = _both_sides(W, 64, nP, sad, geom)
    vol = _vol(W, 64, dtype)
    out = torch.float32 if dtype == "float32" else vol.dtype
    thick = ops.fp_dev(vol, sad, _ang(nP), geom, out_dtype=out, variant=_lib.FP_EXPLICIT)
    for H in (1, 9, H0):
        thin = ops.fp_dev(vol[:H].contiguous(), sad, _ang(nP), geom, out_dtype=out,
                          variant=_lib.FP_EXPLICIT)
        v = _host(vol[:H])
        assert rel_l2(_host(thin), orc.fp(v, sad, _ang(nP), nP, geom)) <= tol
        if dtype == "float32":
            assert rel_l2(_host(thin), _host(thick[:, :H])) <= 2e-6


@pytest.mark.gpu
@pytest.mark.parametrize("geom", [0, 1])
def test_slabs_detectors_and_batches_on_both_sides(cuda, orc, geom):
    """A thin slab of a thick volume, a detector of the volume's own columns, and a batch of
    thin, thick and cone problems agree with the single call: the batch and the detector bit
    for bit."""
    import torch
    from mexct import _lib, batch, ops

    W, H, nP, sad = 70, 64, 150, 300.0
    H0 = _both_sides(W, H, nP, sad, geom)
    ang, vol = _ang(nP), _vol(W, H)
    full = ops.fp_dev(vol, sad, ang, geom, variant=_lib.FP_EXPLICIT)
    total = torch.zeros_like(full)
    for z0, z1 in ((0, 3), (3, 3 + H0), (3 + H0, H)):
        part = vol[z0:z1].contiguous()
        one = ops.fp_sub_dev(part, H, z0, sad, ang, geom)
        assert not one[:, :z0].any() and not one[:, z1:].any()
        ops.fp_sub_dev(part, H, z0, sad, ang, geom, out=total, accumulate=True)
    assert rel_l2(total.cpu().numpy(), full.cpu().numpy()) <= 2e-6
    probs = []
    for g, v in ((geom, vol[:5].contiguous()), (geom, vol), (2, vol[:20].contiguous()),
                 (1 - geom, vol[:H0].contiguous()), (geom, vol)):
        h = v.shape[0]
        det = ops.fp_det_dev(v, sad, ang, g, W, h)
        one = ops.fp_dev(v, sad, ang, g, variant=_lib.FP_EXPLICIT)
        assert torch.equal(det, one)
        probs.append({"vol": v, "sino": torch.zeros((nP, h, W), device="cuda"), "geom": g,
                      "rec": torch.zeros((h, W, W), device="cuda"), "angles": ang, "sad": sad,
                      "want": one})
    b = batch.Batch([{k: p[k] for k in p if k != "want"} for p in probs])
    b.fp()
    torch.cuda.synchronize()
    for p in probs:
        assert torch.equal(p["sino"], p["want"])
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("geom", [0, 1])
@pytest.mark.parametrize("H", [1, 8, 9])
def test_osc_on_both_sides_of_the_rule(cuda, orc, geom, H):
    """15 views of 4 tiles in a subset: the slab kernel up to 8 slices, clusters above."""
    import mexct
    from mexct import tune

    W, nP, nsub, sad = 100, 60, 4, 400.0
    assert tune.fp_plan(W, H, sad, _ang(nP), geom, nsub)[0] == (H > 8)
    rng = np.random.default_rng(H)
    mu = np.asfortranarray(rng.uniform(0, 0.02, (W, W, H)).astype(np.float32))
    pre = np.full((W, H, nP), 1e5, np.float32, order="F")
    post = np.asfortranarray((pre * np.exp(-rng.uniform(0.5, 2, pre.shape))).astype(np.float32))
    picks = np.array([2, 0, 3, 1], np.int32)
    ref = orc.osc_iter(mu, pre, post, nsub, picks, _ang(nP), sad, geom)
    mexct.CUDAmex_oscIter(mu, pre, post, nsub, picks, _ang(nP), sad, geom)
    assert rel_l2(mu, ref) <= 1e-4  # the operator's bound in the parity tests


@pytest.mark.gpu
@pytest.mark.parametrize("geom", ["par3d", "fan3d"])
def test_solvers_of_thin_volumes(cuda, orc, geom):
    """OSC-TV whose iterations run on the slab kernel, with the objective, captured and
    eager, in core and in slabs."""
    import torch
    from mexct import solver, tune

    W, H, nP = 100, 8, 60
    g = {"type": geom, "SAD": 400.0}
    code = 0 if geom == "par3d" else 1
    assert not tune.fp_plan(W, H, 400.0, _ang(nP), code, 4)[0]
    rng = np.random.default_rng(4)
    mu = np.asfortranarray(rng.uniform(0, 0.02, (W, W, H)).astype(np.float32))
    l = orc.osc_fp(mu, 400.0, _ang(nP), code)
    pre = np.full((W, H, nP), 1e5, np.float32, order="F")
    post = np.asfortranarray((pre * np.exp(-l)).astype(np.float32))
    picks = np.array([1, 3], np.int32)
    eager = solver.OSC_TV_recon(pre, post, _ang(nP), g, 2, 0.2, 4, 4, 1.0, picks)
    ref = orc.osc_tv(pre, post, _ang(nP), 400.0, code, 2, 0.2, 4, 4, 1.0, picks)
    assert rel_l2(eager, ref) <= 5e-3  # iterates: the solver tests' bound
    ooc, _ = solver.OSC_TV_recon_ooc(pre, post, _ang(nP), g, 2, 0.2, 4, 4, 1.0, picks, 1 << 34)
    assert rel_l2(ooc, eager) <= 2e-5
    d = [torch.from_numpy(np.ascontiguousarray(a.transpose(2, 1, 0))).cuda() for a in (pre, post)]
    outs = []
    for graph in (False, True):
        s = solver.OscTvSolver(d[0], d[1], _ang(nP), 400.0, code)
        s.run(picks, n_iter=2, tv_const=0.2, n_sub_init=4, n_sub_final=4, p_val=1.0,
              use_graph=graph, objective=True)
        outs.append(s.mu().cpu().numpy().transpose(2, 1, 0))
        obj = s.stats()[2]
        s.close()
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], eager)
    l = orc.osc_fp(outs[1], 400.0, _ang(nP), code)
    p, q = pre.astype(np.float64), post.astype(np.float64)
    p[0, 0, 0] = q[0, 0, 0] = 0.0  # zeroed from iteration 2 on
    want = float(np.sum(p * np.exp(-l) + q * l))
    assert abs(obj - want) <= 1e-6 * abs(want)
