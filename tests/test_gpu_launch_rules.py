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
@pytest.mark.parametrize("form", ["ns", "euler", "fp32", "wale", "learned"])
def test_every_tile_gives_the_same_state(dims, P, n, form):
    visc = form != "euler"
    s = H.Solver.box(dims, P, n, [0.0] * dims, [2 * np.pi] * dims, jitter=0.1, seed=5, viscous=visc,
                     precision=int(form == "fp32"), les=int(form in ("wale", "learned")),
                     sgs_model=5 if form == "learned" else 1, **NS)
    if form == "learned":            # weights that matter: c near softplus(-1)
        w = M.init_params(5)
        w[M.B3] = -1.0
        s.set_sgs_mlp(w)
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


@pytest.mark.parametrize("P,shape", [(1, (3, 1)), (2, (3, 1)), (3, (1, 1))])
def test_mixed_stage_default_shapes(P, shape):
    """Registers for four blocks per SM where more than one fits its shared memory."""
    from hifiles_b200 import mixed as X
    from hifiles_b200 import seam
    xv, c2v = H.box_mesh(3, (3, 3, 2), (0, 0, 0), (1, 1, 1))
    mesh = X.MixedMesh(P, xv, [(X.HEX, tuple(int(v) for v in c)) for c in c2v], np.array([1.0] * 3), (), X.ElementOpts())
    u0 = np.zeros(mesh.types[X.HEX]["pos_upts"].shape[:2] + (5,), order="F")
    u0[..., 0], u0[..., 4] = 1.0, 2.5
    types, ints, bdys = mesh.operator_inputs({X.HEX: u0})
    m = seam.FusedMixedMesh(types, ints, dict(NS, rt_inf=1.0, c_sth=1.0, fix_vis=1.0), bdys)
    assert tuple(m.launch(X.HEX)) == shape


def _box_2d(kind, nx, ny, x1):
    """Vertices and cells of the box [0, x1] x [0, 10], nx x ny quads or pairs of triangles, row by row."""
    from hifiles_b200 import mixed as X
    xv = np.stack([a.ravel() for a in np.meshgrid(np.linspace(0, x1, nx + 1), np.linspace(0, 10, ny + 1))], axis=1)
    cells = []
    for j in range(ny):
        for i in range(nx):
            a, d = i + (nx + 1) * j, i + (nx + 1) * (j + 1)
            if kind == X.QUAD:
                cells.append((X.QUAD, (a, a + 1, d, d + 1)))
            else:
                cells += [(X.TRI, (a, a + 1, d + 1)), (X.TRI, (a, d + 1, d))]
    return xv, cells


# cells of the smaller mesh: at most 4 x 148 elements times 3 blocks per SM
# (Navier-Stokes), 5 (Euler; 10 where a block's elements only double) or 4 (Roe)
@pytest.mark.parametrize("kind,P,form,n", [
    ("tri", 1, "ns", (29, 30)), ("tri", 2, "ns", (29, 30)), ("tri", 3, "ns", (29, 30)), ("tri", 4, "ns", (29, 30)),
    ("tri", 1, "euler", (40, 37)), ("tri", 2, "euler", (40, 37)), ("tri", 3, "euler", (40, 37)),
    ("tri", 4, "euler", (54, 54)), ("tri", 2, "roe", (37, 32)), ("tri", 4, "roe", (37, 32)),
    ("quad", 1, "ns", (42, 42)), ("quad", 2, "ns", (42, 42)), ("quad", 3, "ns", (42, 42)), ("quad", 4, "ns", (42, 42)),
    ("quad", 1, "euler", (54, 54)), ("quad", 2, "euler", (54, 54)), ("quad", 3, "euler", (76, 77)),
    ("quad", 4, "euler", (76, 77)), ("quad", 2, "roe", (48, 49)), ("quad", 3, "roe", (48, 49))])
def test_elements_per_block_do_not_change_the_state(kind, P, form, n):
    """A mesh below the size where the mixed stage's blocks are filled, and two
    copies of it side by side, above: each copy of a periodic state advances as
    the small mesh does.  The copies' coordinates differ from the original's in
    their last bits (20 / 0.13 eps of a cell's size, 4e-14), and so by less than
    1e-12 the states."""
    from hifiles_b200 import mixed as X
    from hifiles_b200 import seam
    t = X.TRI if kind == "tri" else X.QUAD
    cells = n[0] * n[1] * (2 if kind == "tri" else 1)
    most = 4 * 148 * {"ns": 3, "euler": 10 if P >= 4 or (kind == "quad" and P == 3) else 5, "roe": 4}[form]
    assert cells <= most < 2 * cells
    phys = dict(gamma=1.4, prandtl=0.71, mu_inf=1e-2, rt_inf=1.0, c_sth=1.0, fix_vis=1.0, tau=1.0, pen_fact=0.5)
    out = []
    for k in (1, 2):
        xv, c = _box_2d(t, k * n[0], n[1], 10.0 * k)
        mesh = X.MixedMesh(P, xv, c, np.array([10.0 * k, 10.0]), (), X.ElementOpts(vcjh_scheme_tri=1))
        pos = mesh.types[t]["pos_upts"]
        x, y = 0.2 * np.pi * pos[..., 0], 0.2 * np.pi * pos[..., 1]
        rho, u, v = 1 + 0.1 * np.sin(x) * np.cos(y), 0.5 + 0.1 * np.cos(y), 0.2 * np.sin(x + y)
        p = 1 + 0.05 * np.cos(x - y)
        u0 = np.asfortranarray(np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], axis=-1))
        types, ints, bdys = mesh.operator_inputs({t: u0})
        m = seam.FusedMixedMesh(types, ints, phys, bdys, viscous=form == "ns", riemann=2 if form == "roe" else 0)
        nrm = m.advance(3, 1e-3, norms=True)
        out.append((m.get_state(t), nrm, u0))
    (a, na, u0), (b, nb, _) = out
    per = 2 if kind == "tri" else 1
    row = b.reshape(b.shape[0], n[1], 2 * n[0] * per, 4)    # elements row by row
    assert rel(a, u0) > 1e-5 and np.all(np.abs(nb - na) <= 1e-9 * na)
    for copy in (row[:, :, :n[0] * per], row[:, :, n[0] * per:]):
        assert rel(copy.reshape(a.shape), a) <= 1e-12
