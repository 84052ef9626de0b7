"""Kernels that a call takes by its size, on both sides of each line, against the
CPU oracle or the other form."""
import numpy as np
import pytest

from conftest import BULK, EPS0, EPS1, born_case, molecule_case

pytestmark = pytest.mark.gpu


def _solver(case, **kw):
    import tabipb

    kw = dict(dict(order=3, maxparnode=500, theta=0.8, eps0=EPS0, eps1=EPS1,
                   kappa=tabipb.kappa(BULK, EPS1), iprcd=0), **kw)
    s = tabipb.TabiSolver(**kw)
    g = s.form_matrix(case["sptpos"], case["sptnrm"], case["nvert"], case["chrpos"],
                      case["atmchr"])
    s.build_tree()
    return s, g


# far lists below and above 8 M interactions: a mixed handle's items of 64 and of
# 128 targets.  The FP32 sums hold some 1e-6 of cancelling terms (the bar of the
# mixed operator's own tests); the handle's FP64 operator is the FP64 handle's, up
# to the order of each target's sums.
@pytest.mark.parametrize("order", [6, 7, 8])
@pytest.mark.parametrize("level,leaf", [(3, 20), (6, 30)])
def test_mixed_far_items(gpu_lib, order, level, leaf):
    import tabipb

    case = born_case(level, radius=6.0)
    kw = dict(order=order, maxparnode=leaf, theta=0.4 if level > 3 else 0.8, tol=1e-9)
    with _solver(case, **kw)[0] as s:
        n = s.nface
        far = s.counts()[1]
        x = np.random.default_rng(order).normal(size=2 * n)
        y = s.matvec(x)
    with _solver(case, precision=tabipb.PREC_MIXED, **kw)[0] as s:
        assert s.counts()[1] == far
        y32 = s.matvec(x)
    assert (far >= 8 << 20) == (level > 3)
    assert np.linalg.norm(y32 - y) <= 2e-5 * np.linalg.norm(y)


# orders whose Cartesian moments take one or four raw sets per thread: faces times
# terms below and above 400,000
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("level", [2, 4, 5, 6])
def test_mixed_moments(gpu_lib, order, level):
    import tabipb

    case = born_case(level, radius=6.0)
    kw = dict(order=order, maxparnode=20 if level < 5 else 150, theta=0.7)
    y = []
    for prec in (tabipb.PREC_FP64, tabipb.PREC_MIXED):
        with _solver(case, precision=prec, **kw)[0] as s:
            x = np.random.default_rng(order).normal(size=2 * s.nface)
            y.append(s.matvec(x))
    assert np.linalg.norm(y[1] - y[0]) <= 2e-5 * np.linalg.norm(y[0])


@pytest.mark.parametrize("order", [6, 8])
def test_mixed_far_field_in_double(gpu_lib, order):
    """The FP64 residual of a small mixed solve takes one target per thread, the
    FP64 handle's operator two: the mixed solution satisfies the latter."""
    import tabipb

    case = molecule_case(60, 6.0, 2.0, seed=2)
    kw = dict(order=order, maxparnode=100, theta=0.7, iprcd=1, tol=1e-9)
    with _solver(case, precision=tabipb.PREC_MIXED, **kw)[0] as s:
        b = np.random.default_rng(order).normal(size=2 * s.nface)
        r = s.dgmres(b)
    assert r["ierr"] == 0
    with _solver(case, **kw)[0] as s:
        d = s.msolve(b - s.matvec(r["x"]))
        m = s.msolve(b)
    assert np.linalg.norm(d) <= 1.01e-9 * np.linalg.norm(m)


def _near_lists(nodes, xyz, theta):
    """(entries, entries times their leaf's faces, far interactions) of the lists."""
    num, nchild, geo = nodes["numpar"], nodes["nchild"], nodes["geo"]
    at, out = [0], [0, 0, 0]

    def walk(t):  # the nodes come in the order of this walk
        c = at[0]
        at[0] += 1
        far = np.zeros(len(t), bool)
        if num[c] > 40 and len(t):
            far = geo[c, 3] < np.sqrt(((geo[c, :3] - xyz[t]) ** 2).sum(1)) * theta
        out[2] += int(far.sum())
        t = t[~far]
        if nchild[c] == 0:
            out[0] += len(t)
            out[1] += len(t) * int(num[c])
        for _ in range(nchild[c]):
            walk(t)

    walk(np.arange(len(xyz)))
    return out


# threads per target of the FP64 near field (tree.cu, near_split), 1e-12 as in
# test_gpu_matvec_paths.py: sums of the same terms in another order
@pytest.mark.parametrize("level,leaf,theta,split", [
    (3, 20, 0.8, 1), (5, 30, 0.8, 1), (3, 60, 0.7, 2), (5, 150, 0.8, 2), (4, 600, 0.8, 4),
    (1, 7, 0.8, 8), (0, 20, 0.8, 16), (4, 1300, 0.8, 16)])
def test_threads_per_near_target(gpu_lib, level, leaf, theta, split):
    import oracle as O

    case = born_case(level, radius=6.0)
    s, g = _solver(case, maxparnode=leaf, theta=theta)
    with s:
        n, o = s.nface, s.orderarr - 1
        tn, pairs, far = _near_lists(s.tree_nodes(), g[0][o], theta)
        assert (pairs - n, far) == s.counts()
        k = 1
        while k < 16 and tn * k < 148 * 8 * 128 and (pairs >= 16 * k * tn or tn * k < 148 * 128):
            k *= 2
        assert k == split
        x = np.random.default_rng(level).normal(size=2 * n)
        y = s.unpermute(s.matvec(np.concatenate([x[:n][o], x[n:][o]])))
    T = O.Tree(*g, 3, leaf, theta)
    oo = T.orderarr - 1
    yo = T.matvec(O.kappa(BULK, EPS1), EPS1 / EPS0, np.concatenate([x[:n][oo], x[n:][oo]]),
                  nthreads=4)
    ref = np.empty_like(yo)
    ref[oo], ref[n + oo] = yo[:n], yo[n:]
    assert np.linalg.norm(y - ref) <= 1e-12 * np.linalg.norm(ref)


# one leaf around the near field's 256-face tile: a last tile of 255, 1, 44 and 1
# faces, and the target's own face in it
@pytest.mark.parametrize("faces", [255, 256, 257, 300, 513])
def test_near_tiles(gpu_lib, faces):
    import oracle as O

    case = born_case(3, radius=6.0)
    case["nvert"] = np.ascontiguousarray(case["nvert"][:faces])
    s, g = _solver(case, maxparnode=600)
    with s:
        n, o = s.nface, s.orderarr - 1
        assert n == faces and s.leaves()[1].size == 1
        x = np.random.default_rng(faces).normal(size=2 * n)
        y = s.unpermute(s.matvec(np.concatenate([x[:n][o], x[n:][o]])))
    yo = O.matvec_direct(*g[:3], O.kappa(BULK, EPS1), EPS1 / EPS0, x)
    assert np.linalg.norm(y - yo) <= 1e-12 * np.linalg.norm(yo)


# blocks around the unpivoted factorisation's 16, 32, 64 and 128 columns: certified,
# so the edges tested are its own and not the pivoted kernels'
@pytest.mark.parametrize("faces", [2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 97, 129, 193,
                                   320])
def test_edges_are_certified(gpu_lib, faces):
    import oracle as O

    kappa = O.kappa(BULK, EPS1)
    case = born_case(2, radius=3.0)
    case["nvert"] = np.ascontiguousarray(case["nvert"][:faces])
    s, g = _solver(case, iprcd=1, kappa=kappa)
    with s:
        n, o = s.nface, s.orderarr - 1
        assert n == faces and s.pivoted_leaves() == 0
        r = np.random.default_rng(faces).normal(size=2 * n)
        z = s.unpermute(s.msolve(np.concatenate([r[:n][o], r[n:][o]])))
    T = O.Tree(*g, 3, 500, 0.8)
    oo = T.orderarr - 1
    zt = T.msolve(kappa, EPS1 / EPS0, np.concatenate([r[:n][oo], r[n:][oo]]))
    zo = np.empty_like(zt)
    zo[oo], zo[n + oo] = zt[:n], zt[n:]
    assert np.linalg.norm(z - zo) <= 1e-10 * np.linalg.norm(zo)


# the network's products in column blocks of 64 (80 blocks of 64 panels) and of all or
# half the columns (320); blocks of 32 are test_gpu_kernel_edges.py's.  Bars as there.
@pytest.mark.parametrize("level,hidden", [(4, 32), (4, 96), (4, 160), (4, 256), (5, 32), (5, 96),
                                          (5, 160), (5, 224)])
def test_network_products(gpu_lib, level, hidden):
    import torch
    import warmstart_ref as W

    import oracle as O
    from tabipb.warmstart import WarmStart

    c = born_case(level, radius=3.0)
    xyz, tq, ar, b = O.form_matrix(c["sptpos"], c["sptnrm"], c["nvert"], c["chrpos"] + 0.4,
                                   c["atmchr"], 1.0)
    rng = np.random.default_rng(hidden)
    x = b * 0.3 + rng.standard_normal(b.size) * np.std(b) * 0.1
    z = b * 0.25 + rng.standard_normal(b.size) * np.std(b) * 0.05
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64).ravel()).cuda()
    s = dict(n=len(ar), xyz=t(xyz), tq=t(tq), area=t(ar), b=t(b), z=t(z), x=t(x))
    ws = WarmStart(hidden=hidden, layers=1, seed=0)
    theta = W.init_params(hidden, 1, 8, seed=4)
    ws.set_params(theta)
    nbr = ws.graph_dev(s)[0].astype(np.int64)
    xr, loss_ref, cache = W.forward(theta, hidden, 1, 8, xyz.reshape(-1, 3), tq.reshape(-1, 3), ar,
                                    b, nbr, target=x, z=z)
    g_ref = W.backward(cache, hidden, 1, 8, nbr)
    loss, g = ws.loss_grad_dev(s)
    assert abs(loss - loss_ref) <= 1e-4 * abs(loss_ref)
    o = 0
    for name, shp in W.param_shapes(hidden, 1, 8):
        k = int(np.prod(shp))
        d = np.abs(g[o:o + k] - g_ref[o:o + k]).max()
        assert d <= 2e-3 * (np.abs(g_ref[o:o + k]).max() + 1e-30), name
        o += k
    xp = torch.empty_like(s["b"])
    ws.predict_dev(s, xp)
    assert np.linalg.norm(xp.cpu().numpy() - xr) <= 5e-4 * np.linalg.norm(xr)


# one block of order > 512: the row form (factors up to 56 MiB, or an odd number of
# faces up to order 7,500) and the streamed one, full and partial last steps.  B z = r
# with B as LEAFMATVECpara assembles it, as in test_gpu_kernel_edges.py.
@pytest.mark.parametrize("faces", [257, 272, 399, 416, 1354, 1356, 1447, 1448, 1450, 1456, 3749, 3751])
def test_forms_of_the_block_apply(gpu_lib, faces):
    kappa, eps = 0.1257, EPS1 / EPS0
    case = born_case(4, radius=6.0)
    case["nvert"] = np.ascontiguousarray(case["nvert"][:faces])
    s, g = _solver(case, kappa=kappa, iprcd=1, maxparnode=4000)
    with s:
        n, o = s.nface, s.orderarr - 1
        assert n == faces and s.leaves()[1].size == 1
        r = np.random.default_rng(faces).normal(size=2 * n)
        z = s.msolve(r)
        xyz, nrm, ar = (np.asarray(v).reshape(n, -1)[o] for v in g[:3])
    for i in range(0, n, 500):
        j = min(n, i + 500)
        d = xyz[None] - xyz[i:j, None]
        rs = np.sqrt((d ** 2).sum(-1))
        own = rs == 0
        rs[own] = 1.0
        g0, e = 1 / (4 * np.pi * rs), np.exp(-kappa * rs)
        v, v0 = nrm[None], nrm[i:j, None]
        c, c0, vv = (v * d).sum(-1) / rs, (v0 * d).sum(-1) / rs, (v * v0).sum(-1)
        t1, t2 = g0 / rs, (1 + kappa * rs) * e
        g3 = (vv - 3 * c0 * c) / rs * t1
        k1, k2 = c * t1 * (1 - eps * t2), g0 * (1 - e)
        k3, k4 = g3 * (t2 - 1) - kappa ** 2 * c0 * c * e * g0, c0 * t1 * (1 - t2 / eps)
        a = np.where(own, 0.0, ar.ravel()[None])
        y1 = .5 * (1 + eps) * z[i:j] - (k1 * a) @ z[:n] - (k3 * a) @ z[n:]
        y2 = .5 * (1 + 1 / eps) * z[n + i:n + j] - (k2 * a) @ z[:n] - (k4 * a) @ z[n:]
        assert np.abs(y1 - r[i:j]).max() <= 1e-10
        assert np.abs(y2 - r[n + i:n + j]).max() <= 1e-10
