"""Launch rules of the stage, closure and mixed-mesh kernels at the sizes where
they can go wrong: tail blocks, meshes smaller than one block, several tiles
per persistent block, block counts that are not a power of two.

States are compared bit for bit (a launch shape changes no element's
arithmetic).  Norms are sums of positive terms in another order: n terms give
at most n eps relative, 1e-12 for the 10^3 block sums here."""
import numpy as np
import pytest

import hifiles_b200 as H
import mlp as M
import oracle as O
from golden_util import rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NS = dict(gamma=1.4, prandtl=0.71, mu_inf=1e-3, tau=1.0, pen_fact=0.5)


@pytest.mark.parametrize("dims,P,n", [(2, 1, (5, 7)), (2, 2, (3, 7)), (2, 3, (5, 5)), (2, 4, (7, 3)), (2, 5, (3, 5)),
                                      (3, 1, (3, 5, 3)), (3, 2, (3, 3, 3)), (3, 3, (1, 3, 1)), (3, 4, (1, 1, 1)),
                                      (3, 4, (3, 1, 3))])
@pytest.mark.parametrize("form", ["ns", "euler", "fp32", "wale"])
def test_every_tile_gives_the_same_state(dims, P, n, form):
    visc = form != "euler"
    s = H.Solver.box(dims, P, n, [0.0] * dims, [2 * np.pi] * dims, jitter=0.1, seed=5, viscous=visc,
                     precision=int(form == "fp32"), les=int(form == "wale"), sgs_model=1, **NS)
    pos = s.geometry()["pos_upts"]
    u0 = O.ic_tgv(pos) if dims == 3 else O.ic_vortex(pos * (10 / (2 * np.pi)) - 5)
    s.set_state(u0)
    s.advance(2, 1e-4)               # the tiles chosen for this mesh
    ref = s.get_state()
    assert np.isfinite(ref).all() and not np.array_equal(ref, u0)
    ng, nu = s.tile_count()
    for g, u in [(g, 0) for g in range(ng)] + [(0, u) for u in range(1, nu)]:
        s.set_state(u0)
        s.select_tiles(g, u)
        s.advance(2, 1e-4)
        assert np.array_equal(s.get_state(), ref), (s.tile_info(0, g), s.tile_info(1, u))


@pytest.mark.parametrize("n", [1, 127, 129, 128 * 296 + 5, 128 * 600 - 1])
def test_closure_gradient_at_tile_edges(n):
    """Less than a tile, one more than a tile, and one or two tiles per persistent block."""
    rng = np.random.default_rng(n)
    w = M.init_params(3, xmean=rng.normal(0, 0.2, 6).astype(np.float32),
                      xscale=rng.uniform(0.5, 2.0, 6).astype(np.float32))
    X, Y = rng.standard_normal((n, 6)).astype(np.float32), rng.uniform(0.0, 0.5, n).astype(np.float32)
    sw = rng.uniform(0.0, 3.0, n).astype(np.float32)
    dev = [torch.from_numpy(a).cuda() for a in (w, X, Y, sw)]
    g = torch.empty(H.mlp_n_trained(), dtype=torch.float32, device="cuda")
    loss = torch.empty(1, dtype=torch.float32, device="cuda")
    ns = H.mlp_scratch_floats(n)
    scratch = torch.empty(ns, dtype=torch.float32, device="cuda")
    H.mlp_loss_grad(dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), n, g.data_ptr(), loss.data_ptr(),
                    scratch.data_ptr(), ns, d_sw=dev[3].data_ptr())
    torch.cuda.synchronize()
    l_ref, g_ref = M.loss_grad(w, X, Y, sw)
    assert abs(loss.item() - l_ref) <= 1e-5 * l_ref
    assert rel(g.cpu().numpy(), g_ref) < 1e-4


@pytest.mark.parametrize("n", [129, 128 * 295 + 1, 128 * 296 + 1, 128 * 700])
def test_closure_gradient_partials_depend_on_the_batch_alone(n):
    """One partial gradient per tile of 128 samples, 296 at most whatever the
    GPU's number of SMs: their number decides a gradient's last bits."""
    rng = np.random.default_rng(n)
    dev = [torch.from_numpy(a.astype(np.float32)).cuda()
           for a in (M.init_params(3), rng.standard_normal((n, 6)), rng.uniform(0.0, 0.5, n))]
    g = torch.empty(H.mlp_n_trained(), dtype=torch.float32, device="cuda")
    loss = torch.empty(1, dtype=torch.float32, device="cuda")
    ns = H.mlp_scratch_floats(n)
    scratch = torch.full((ns,), float("nan"), dtype=torch.float32, device="cuda")
    H.mlp_loss_grad(dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), n, g.data_ptr(), loss.data_ptr(),
                    scratch.data_ptr(), ns)
    torch.cuda.synchronize()
    used = min(-(-n // 128), 296) * (H.mlp_n_trained() + 1)
    assert bool(torch.isfinite(scratch[:used]).all()) and bool(torch.isnan(scratch[used:]).all())


@pytest.mark.parametrize("P,viscous", [(1, False), (2, False), (3, True)])
def test_mixed_norms_do_not_depend_on_the_launch_shape(P, viscous):
    """6498 triangles: more block sums than the 256 threads that add them in
    every shape, and a tail block.  At dt 1e-12 the last stage's residual is that
    of the initial state: the state moves by 1e-12 of its residual, and the
    residual of a small change is at most some wave speeds times the squared
    order over the spacing (10 x 16 / 0.175, under 1e3) times that change, so
    1e-9 of it; a lost block sum would be a thousandth."""
    from hifiles_b200 import mixed as X
    from hifiles_b200 import seam
    from test_gpu_order_tri import EULER, tri_box
    xv, tris = tri_box(57)
    mesh = X.MixedMesh(P, xv, [(X.TRI, t) for t in tris], [10.0, 10.0], [], X.ElementOpts(vcjh_scheme_tri=1))
    u0 = np.asfortranarray(O.ic_vortex(mesh.types[X.TRI]["pos_upts"]))
    types, ints, bdys = mesh.operator_inputs({X.TRI: u0})
    ph = dict(EULER, mu_inf=1e-3, tau=1.0) if viscous else EULER
    still = seam.FusedMixedMesh(types, ints, ph, bdys, viscous=viscous)
    still.residual()
    div = still.S[X.TRI]["div"].cpu().numpy().reshape(u0.shape, order="F")
    want = np.abs(div / np.asarray(types[X.TRI]["detjac_upts"])[:, :, None]).mean(axis=(0, 1))
    assert np.all(want > 0)
    out = []
    for g, u in ((0, 0), (1, 1), (3, 2), (4, 1)) if viscous else ((1, 1),):
        m0 = seam.FusedMixedMesh(types, ints, ph, bdys, viscous=viscous)
        m0.set_launch(X.TRI, g, u)
        nrm = m0.advance(1, 1e-12, norms=True)
        assert np.all(np.abs(nrm - want) <= 1e-9 * want), (g, u, nrm, want)
        m = seam.FusedMixedMesh(types, ints, ph, bdys, viscous=viscous)
        m.set_launch(X.TRI, g, u)
        nrm = m.advance(2, 1e-3, norms=True)
        # the same two steps without norms leave the same state
        m2 = seam.FusedMixedMesh(types, ints, ph, bdys, viscous=viscous)
        m2.advance(2, 1e-3)
        out.append((nrm, m.get_state(X.TRI)))
        assert np.array_equal(out[-1][1], m2.get_state(X.TRI))
    for nrm, st in out:
        assert np.all(nrm > 0) and np.array_equal(st, out[0][1])
        assert np.all(np.abs(nrm - out[0][0]) <= 1e-12 * out[0][0])
