"""Values at the edges of the solver's arithmetic: pivots whose reciprocal is
subnormal, atoms on a face's centroid, gates far below zero, and the rounding tie
that decides on a second orthogonalisation."""
import ctypes as C

import numpy as np
import pytest

from conftest import BULK, EPS0, EPS1, born_case

pytestmark = pytest.mark.gpu


def _kappa():
    import tabipb

    return tabipb.kappa(BULK, EPS1)


def test_pivots_above_the_reciprocal(gpu_lib):
    """A dielectric ratio of 1e308: the diagonal of the blocks' first half is
    5e307, whose reciprocal is subnormal.  B z = r with B as LEAFMATVECpara
    assembles it; the subnormal reciprocals (1e-308, to 5e-324) leave 1e-13."""
    import tabipb

    kappa, eps = 0.1257, 1e308
    case = born_case(1, radius=3.0)
    with tabipb.TabiSolver(order=3, maxparnode=100, theta=0.8, eps0=1.0, eps1=eps, kappa=kappa,
                           iprcd=1) as s:
        xyz, nrm, ar, _ = s.form_matrix(case["sptpos"], case["sptnrm"], case["nvert"],
                                        case["chrpos"], case["atmchr"])
        s.build_tree()
        n, o = s.nface, s.orderarr - 1
        assert s.leaves()[1].size == 1
        r = np.random.default_rng(1).normal(size=2 * n)
        r[:n] *= 1e300
        z = s.msolve(r)
    xyz, nrm, ar = xyz[o], nrm[o], ar[o]
    d = xyz[None] - xyz[:, None]
    rs = np.sqrt((d ** 2).sum(-1))
    own = rs == 0
    rs[own] = 1.0
    g0, e = 1 / (4 * np.pi * rs), np.exp(-kappa * rs)
    c, c0 = (nrm[None] * d).sum(-1) / rs, (nrm[:, None] * d).sum(-1) / rs
    t1, t2 = g0 / rs, (1 + kappa * rs) * e
    g3 = (nrm @ nrm.T - 3 * c0 * c) / rs * t1
    a = np.where(own, 0.0, ar[None])
    k1, k2 = c * t1 * (1 - eps * t2) * a, g0 * (1 - e) * a
    k3 = (g3 * (t2 - 1) - kappa ** 2 * c0 * c * e * g0) * a
    k4 = c0 * t1 * (1 - t2 / eps) * a
    y1 = .5 * (1 + eps) * z[:n] - k1 @ z[:n] - k3 @ z[n:]
    y2 = .5 * (1 + 1 / eps) * z[n:] - k2 @ z[:n] - k4 @ z[n:]
    assert np.abs(y1 - r[:n]).max() <= 1e-10 * 1e300
    assert np.abs(y2 - r[n:]).max() <= 1e-10


@pytest.mark.parametrize("charge", [1.5, -1.5])
def test_atom_on_a_centroid(gpu_lib, charge):
    """1/|d| is infinite for the face whose centroid is the atom's place, and
    that face alone: its potential half is +-Inf, its field half (0 * Inf) NaN,
    from tabi_form_matrix and tabi_rhs alike."""
    import tabipb

    case = born_case(2, radius=3.0)
    # more atoms than one staged tile, the one on the centroid in the second
    chrpos = np.random.default_rng(0).normal(size=(700, 3)) * 0.3
    q = np.full(700, 0.01)
    args = case["sptpos"], case["sptnrm"], case["nvert"]
    with tabipb.TabiSolver(order=3, maxparnode=100, theta=0.8, eps0=EPS0, eps1=EPS1,
                           kappa=_kappa()) as s:
        xyz, _, _, b0 = s.form_matrix(*args, chrpos, q)
        n, k = s.nface, 77
        chrpos[600], q[600] = xyz[k], charge
        b = s.form_matrix(*args, chrpos, q)[3]
        rhs = s.rhs(chrpos, q)
    assert np.isfinite(b0).all()
    for v in (b, rhs):
        assert v[k] == np.copysign(np.inf, charge) and np.isnan(v[n + k])
        rest = np.delete(v, [k, n + k])
        assert np.isfinite(rest).all()


@pytest.mark.parametrize("x", [-87.0, -87.5, -88.0, -88.6, -88.8, -95.0])
def test_gate_far_below_zero(gpu_lib, x):
    """silu(x) for x around -ln(FLT_MAX), where the sigmoid is subnormal: the
    input layer's output, with zero message-passing layers, times 1e36.  The
    exponential's argument is rounded to 2^-24 of 88 (5e-6 of its value), the
    subnormal quotient to 2^-149 (4e-7 of 3e-39); e^88.73 and above overflows
    and gives 0."""
    import torch
    import warmstart_ref as W

    from tabipb.warmstart import WarmStart

    hidden = 32
    theta = {n: np.zeros(s, np.float32) for n, s in W.param_shapes(hidden, 1, 8)}
    theta["b0"][:] = x
    theta["Wo"][:, 0] = 1e36
    ws = WarmStart(hidden=hidden, layers=1, seed=0)
    ws.set_params(np.concatenate([theta[n].ravel() for n, _ in W.param_shapes(hidden, 1, 8)]))
    import oracle as O

    c = born_case(1, radius=3.0)
    xyz, tq, ar, b = O.form_matrix(c["sptpos"], c["sptnrm"], c["nvert"], c["chrpos"] + 0.4,
                                   c["atmchr"], 1.0)
    n = len(ar)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64).ravel()).cuda()
    s = dict(n=n, xyz=t(xyz), tq=t(tq), area=t(ar), b=t(b), z=t(0 * b), x=t(b))
    out = torch.empty_like(s["b"])
    ws.predict_dev(s, out)
    out = out.cpu().numpy()[:n] / np.sqrt(np.mean(b[:n] ** 2))
    wo = float(W.bf16_round(np.float32([1e36]))[0])
    want = hidden * wo * x / (1.0 + np.exp(-float(np.float32(x))))
    if x < -88.73:
        want = 0.0
    assert np.abs(out - want).max() <= 1e-4 * abs(want)


def test_second_orthogonalisation_at_the_tie(gpu_lib):
    """The second step's vector in a Krylov space made by the exchange hook, with
    0.001 * |w| a double on the rounding tie of |v| + 0.001 |w| == |v|, while the
    unrounded product lies above it: the test is DORTH's, each operation rounded,
    and all of the step follows one answer."""
    import tabipb

    s0 = float.fromhex("0x1.f4p-44")  # 0.001 * s0 rounds to 2^-53
    assert 0.001 * s0 == 2.0 ** -53 and np.sqrt(s0 * s0) == s0
    rt = C.CDLL("libcudart.so.12")
    rt.cudaStreamSynchronize.argtypes = [C.c_void_p]
    rt.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    case = born_case(1)
    calls = []
    with tabipb.TabiSolver(order=3, maxparnode=40, theta=0.8, eps0=EPS0, eps1=EPS1,
                           kappa=_kappa(), iprcd=0, tol=0.0, maxl=2, nrmax=-1) as s:
        s.form_matrix(case["sptpos"], case["sptnrm"], case["nvert"], case["chrpos"],
                      case["atmchr"])
        s.build_tree()
        n = s.nface
        # M^-1 b, then A V1, M^-1 A V1, A V2, M^-1 A V2
        heads = [[1.0], [0.0], [1.0, s0], [0.0], [0.3, 0.5, 0.4]]

        def exchange(v, n2, t0, t1, stream):
            w = np.zeros(n2)
            w[:len(heads[len(calls)])] = heads[len(calls)]
            calls.append(n2)
            assert rt.cudaStreamSynchronize(stream) == 0
            assert rt.cudaMemcpy(v, w.ctypes.data, w.nbytes, 1) == 0

        s.set_target_range(0, int(s.leaves()[1][0]))
        s.set_exchange(exchange)
        res = s.dgmres(np.ones(2 * n))
        s.set_exchange(None)
    assert len(calls) == len(heads) and s.exchange_error is None
    # |e1 - H y| over the two columns of H
    h1, h2 = np.array([1.0, s0, 0.0]), np.array([0.3, 0.5, 0.4])
    nrm = np.cross(h1, h2)
    want = [s0, abs(nrm[0]) / np.linalg.norm(nrm)]
    np.testing.assert_allclose(res["err_hist"], want, rtol=1e-9)
    assert res["iter"] == 2 and res["ierr"] == 1
