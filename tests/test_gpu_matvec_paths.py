"""The FP64 operator's kernels against the CPU oracle where they can go wrong:
every Taylor order of the harmonic far field, several screening lengths (zero,
the physiological one, and ones whose exponentials leave the near field's
table), and sizes that take each number of threads per near-field target.

Bar: both sides evaluate the same sums in FP64 in another order; with terms of
both signs cancelling to a few per cent of their magnitude, 1e-12 relative L2
is a few thousand ulp.
"""
import numpy as np
import pytest

from conftest import EPS0, EPS1, born_case, molecule_case

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _compare(case, kappa, order=3, maxparnode=100, theta=0.8):
    import oracle as O
    import tabipb

    with tabipb.TabiSolver(order=order, maxparnode=maxparnode, theta=theta, kappa=kappa,
                           eps0=EPS0, eps1=EPS1, iprcd=0) as s:
        xyz, tq, ar, b = s.form_matrix(case["sptpos"], case["sptnrm"], case["nvert"],
                                       case["chrpos"], case["atmchr"])
        T = O.Tree(xyz, tq, ar, b, order, maxparnode, theta)
        oa, _ = s.build_tree()
        n = len(ar)
        x = np.random.default_rng(order).normal(size=2 * n)
        o = oa - 1
        y = s.unpermute(s.matvec(np.concatenate([x[:n][o], x[n:][o]])))
        oo = T.orderarr - 1
        yo = T.matvec(kappa, EPS1 / EPS0, np.concatenate([x[:n][oo], x[n:][oo]]))
        ref = np.empty_like(yo)
        ref[oo], ref[n + oo] = yo[:n], yo[n:]
    assert np.linalg.norm(y - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("kappa", [0.0, 0.1257, 2.5])
@pytest.mark.parametrize("order", range(1, 9))
def test_orders(gpu_lib, order, kappa):
    _compare(born_case(3), kappa, order=order, maxparnode=60, theta=0.7)


# 20 faces (one leaf, no far field) to 20,480; leaves below and above the
# near field's 512-face tile and off its multiples
@pytest.mark.parametrize("level,leaf", [(0, 20), (1, 7), (2, 33), (3, 1280), (4, 600), (5, 150)])
def test_sizes(gpu_lib, level, leaf):
    _compare(born_case(level, radius=6.0), 0.1257, maxparnode=leaf)


@pytest.mark.parametrize("kappa", [1.0, 40.0])
def test_screened_molecule(gpu_lib, kappa):
    _compare(molecule_case(60, 6.0, 2.0, seed=3), kappa, order=4, maxparnode=150)
