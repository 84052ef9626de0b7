"""Kernels at the edges of their tiles and dispatch rules: leaf blocks around
multiples of the factorisation's 16, 64 and 128 columns, every hidden width of
the warm-start network, every order of the mixed far field, exponentials below
the table's end in assembly and energy, the solver's second orthogonalisation,
and handles that reuse memory of earlier ones from several threads.

Bars: preconditioner applies 1e-10 (condition numbers of leaf blocks, a few
hundred, times the rounding of an LU of up to 640 rows); the FP32 operator and
the network as in their own tests; energies 1e-11 (sums in FP64 in another
order, cancellation up to 1e3); reused memory changes no bit.
"""
import threading

import numpy as np
import pytest

from conftest import BULK, EPS0, EPS1, born_case, molecule_case

pytestmark = pytest.mark.gpu


def _handle(case, **kw):
    import tabipb

    kw = dict(dict(order=3, maxparnode=500, theta=0.8, eps0=EPS0, eps1=EPS1,
                   kappa=tabipb.kappa(BULK, EPS1)), **kw)
    s = tabipb.TabiSolver(**kw)
    g = s.form_matrix(case["sptpos"], case["sptnrm"], case["nvert"], case["chrpos"],
                      case["atmchr"])
    s.build_tree()
    return s, g


def _tree(case, order=3, maxparnode=500, theta=0.8):
    import oracle as O

    g = O.form_matrix(case["sptpos"], case["sptnrm"], case["nvert"], case["chrpos"],
                      case["atmchr"], EPS0)
    return O.Tree(*g, order, maxparnode, theta)


def _order(v, o, n):
    return np.concatenate([v[:n][o - 1], v[n:][o - 1]])


def _unorder(v, o, n):
    r = np.empty_like(v)
    r[o - 1], r[n + o - 1] = v[:n], v[n:]
    return r


# one leaf of k faces (a block of order 2k), kappa inside and outside the table
@pytest.mark.parametrize("kappa", [0.1257, 30.0])
@pytest.mark.parametrize("faces", [2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 95, 97, 127, 128, 129,
                                   161, 191, 193, 320])
def test_leaf_block(gpu_lib, faces, kappa):
    case = born_case(2, radius=3.0)
    case["nvert"] = np.ascontiguousarray(case["nvert"][:faces])
    s, _ = _handle(case, kappa=kappa, iprcd=1)
    with s:
        T = _tree(case)
        n = s.nface
        assert n == faces
        r = np.random.default_rng(faces).normal(size=2 * n)
        z = _unorder(s.msolve(_order(r, s.orderarr, n)), s.orderarr, n)
        zo = _unorder(T.msolve(kappa, EPS1 / EPS0, _order(r, T.orderarr, n)), T.orderarr, n)
    assert np.linalg.norm(z - zo) <= 1e-10 * np.linalg.norm(zo)


def test_huge_leaf_block(gpu_lib):
    """One block of order 7,000 (above the apply's 6,912): B z = r, with B as
    LEAFMATVECpara assembles it."""
    kappa, eps = 0.1257, EPS1 / EPS0
    case = born_case(4, radius=6.0)
    case["nvert"] = np.ascontiguousarray(case["nvert"][:3500])
    s, g = _handle(case, kappa=kappa, iprcd=1, maxparnode=4000)
    with s:
        n, o = s.nface, s.orderarr - 1
        assert n == 3500 and s.leaves()[1].size == 1
        r = np.random.default_rng(9).normal(size=2 * n)
        z = s.msolve(r)
        xyz, nrm, ar = (np.asarray(v).reshape(len(s.orderarr), -1)[o] for v in g[:3])
    for i in range(0, n, 500):
        d = xyz[None] - xyz[i:i + 500, None]
        rs = np.sqrt((d ** 2).sum(-1))
        own = rs == 0
        rs[own] = 1.0
        g0, e = 1 / (4 * np.pi * rs), np.exp(-kappa * rs)
        v, v0 = nrm[None], nrm[i:i + 500, None]
        c, c0, vv = (v * d).sum(-1) / rs, (v0 * d).sum(-1) / rs, (v * v0).sum(-1)
        t1, t2 = g0 / rs, (1 + kappa * rs) * e
        g3 = (vv - 3 * c0 * c) / rs * t1
        k1, k2 = c * t1 * (1 - eps * t2), g0 * (1 - e)
        k3, k4 = g3 * (t2 - 1) - kappa ** 2 * c0 * c * e * g0, c0 * t1 * (1 - t2 / eps)
        a = np.where(own, 0.0, ar.ravel()[None])
        y1 = .5 * (1 + eps) * z[i:i + 500] - (k1 * a) @ z[:n] - (k3 * a) @ z[n:]
        y2 = .5 * (1 + 1 / eps) * z[n + i:n + i + 500] - (k2 * a) @ z[:n] - (k4 * a) @ z[n:]
        assert np.abs(y1 - r[i:i + 500]).max() <= 1e-10
        assert np.abs(y2 - r[n + i:n + i + 500]).max() <= 1e-10


@pytest.mark.parametrize("order", range(1, 9))
def test_mixed_orders(gpu_lib, order):
    import tabipb

    case = molecule_case(60, 6.0, 2.0, seed=2)
    y = []
    for prec in (tabipb.PREC_FP64, tabipb.PREC_MIXED):
        s, _ = _handle(case, order=order, maxparnode=100, theta=0.7, precision=prec)
        with s:
            x = np.random.default_rng(order).normal(size=2 * s.nface)
            y.append(s.matvec(x))
    assert np.linalg.norm(y[1] - y[0]) <= 2e-5 * np.linalg.norm(y[0])


@pytest.mark.parametrize("kappa", [0.0, 0.1257, 30.0])
def test_energy(gpu_lib, kappa):
    case = molecule_case(61, 6.0, 2.0, seed=5)
    s, g = _handle(case, kappa=kappa)
    with s:
        n = s.nface
        x = np.random.default_rng(1).normal(size=2 * n) + 2.0
        e, _ = s.energy(case["chrpos"], case["atmchr"], _order(x, s.orderarr, n))
        T = _tree(case)
        eo, _ = T.energy(case["chrpos"], case["atmchr"], kappa, EPS1 / EPS0, EPS0,
                         _order(x, T.orderarr, n))
    assert abs(e - eo) <= 1e-11 * abs(eo)


@pytest.mark.parametrize("level,steps", [(0, 2), (1, 4)])
def test_second_orthogonalisation(gpu_lib, level, steps):
    """A charge at the centre of an icosphere: the Krylov space is that of the
    panels' orbits under the sphere's rotations (one or two), and the step that
    exhausts it leaves rounding only, which asks for a second orthogonalisation."""
    import oracle as O

    case = born_case(level)
    kap = O.kappa(BULK, EPS1)
    s, g = _handle(case, iprcd=0, tol=1e-10)
    with s:
        n = s.nface
        res = s.dgmres(_order(g[3], s.orderarr, n))
        T = _tree(case)
        ref = T.dgmres(kap, EPS1 / EPS0, T.bvct, iprcd=0, tol=1e-10)
        assert res["ierr"] == ref["ierr"] == 0 and res["iter"] == ref["iter"] == steps
        x, xo = _unorder(res["x"], s.orderarr, n), _unorder(ref["x"], T.orderarr, n)
    assert np.linalg.norm(x - xo) <= 1e-9 * np.linalg.norm(xo)


@pytest.mark.parametrize("hidden", [32, 64, 96, 128, 160, 192, 224, 256])
def test_network_widths(gpu_lib, hidden):
    import torch
    import warmstart_ref as W

    import oracle as O
    from tabipb.warmstart import WarmStart

    c = born_case(2, radius=3.0)
    xyz, tq, ar, b = O.form_matrix(c["sptpos"], c["sptnrm"], c["nvert"], c["chrpos"] + 0.4,
                                   c["atmchr"], 1.0)
    rng = np.random.default_rng(hidden)
    x = b * 0.3 + rng.standard_normal(b.size) * np.std(b) * 0.1
    z = b * 0.25 + rng.standard_normal(b.size) * np.std(b) * 0.05
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64).ravel()).cuda()
    s = dict(n=len(ar), xyz=t(xyz), tq=t(tq), area=t(ar), b=t(b), z=t(z), x=t(x))
    ws = WarmStart(hidden=hidden, layers=2, seed=0)
    theta = W.init_params(hidden, 2, 8, seed=4)
    ws.set_params(theta)
    nbr = ws.graph_dev(s)[0].astype(np.int64)
    xr, loss_ref, cache = W.forward(theta, hidden, 2, 8, xyz.reshape(-1, 3), tq.reshape(-1, 3), ar,
                                    b, nbr, target=x, z=z)
    g_ref = W.backward(cache, hidden, 2, 8, nbr)
    loss, g = ws.loss_grad_dev(s)
    assert abs(loss - loss_ref) <= 1e-4 * abs(loss_ref)
    o = 0
    for name, shp in W.param_shapes(hidden, 2, 8):
        k = int(np.prod(shp))
        d = np.abs(g[o:o + k] - g_ref[o:o + k]).max()
        assert d <= 2e-3 * (np.abs(g_ref[o:o + k]).max() + 1e-30), name
        o += k
    xp = torch.empty_like(s["b"])
    ws.predict_dev(s, xp)
    assert np.linalg.norm(xp.cpu().numpy() - xr) <= 5e-4 * np.linalg.norm(xr)


def test_reused_memory(gpu_lib):
    """Handles made and closed in turn, in three threads at once, on molecules
    of different sizes: every solve has the bits of the first."""
    cases = [molecule_case(n, 3.0 + n / 20, 2.0, seed=n) for n in (5, 30, 60)]

    def solve(case):
        s, g = _handle(case, maxparnode=150, iprcd=1)
        with s:
            res = s.dgmres(_order(g[3], s.orderarr, s.nface))
            return res["x"], s.energy(case["chrpos"], case["atmchr"], res["x"])[0]

    want = [solve(c) for c in cases]
    bad = []

    def work(k):
        try:
            for i in range(6):
                j = (i + k) % 3
                x, e = solve(cases[j])
                if not np.array_equal(x, want[j][0]) or e != want[j][1]:
                    bad.append((k, i))
        except Exception as err:  # a thread's error must reach the test
            bad.append(repr(err))

    th = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
