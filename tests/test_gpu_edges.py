"""Calls at the edges of what the entry points accept: targets anywhere, memory of
any alignment and kind, applies that are never evaluated, repeated calls."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]

EPS = 2.0 ** -52


def cloud(n, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.standard_normal(n)


def fmm(kind, k, x, y, cutoff, iscomplex=False, nequiv=24, **kw):
    import pykifmm2d_b200 as P
    kern = {"laplace": lambda k: P.LaplaceKernel(), "k0": P.ModifiedHelmholtzKernel, "h0": P.HelmholtzKernel}[kind](k)
    f = P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), nequiv, cutoff, iscomplex,
              **kw)
    f.build_tree()
    f.precompute()
    return f


@pytest.mark.parametrize("kind,k,iscomplex,precision", [
    ("laplace", 0.0, False, "fp64"), ("laplace", 0.0, True, "fp64"), ("laplace", 0.0, False, "mixed"),
    ("k0", 2.0, False, "fp64"), ("k0", 60.0, False, "fp64"), ("k0", 2.0, False, "mixed"), ("h0", 2.0, True, "fp64")])
def test_targets_anywhere(kind, k, iscomplex, precision):
    """A target that is not a number has no potential; the logarithm at infinity, or
    where r^2 overflows, is infinite (a sum of both signs: not a number), and K0 and
    H0 vanish there.  Targets beside them in the same leaf keep their values: the
    same sums, split over the lanes in another way."""
    x, y, tau = cloud(3000, 3)
    f = fmm(kind, k, x, y, 40, iscomplex, precision=precision)
    f.build_expansions(tau + 0j if iscomplex else tau)
    fx, fy, _ = cloud(500, 4)
    ref = f.evaluate_to_points(fx, fy, False)
    nan, inf, big = np.nan, np.inf, 1e200
    odd = np.array([(nan, 0.1), (-nan, 0.1), (0.1, nan), (nan, nan), (inf, 0.2), (-inf, 0.2), (0.2, inf), (-inf, inf),
                    (big, 0.0), (0.0, -big), (-big, big), (2e154, 0.5)])
    tx, ty = np.concatenate([odd[:, 0], fx]), np.concatenate([odd[:, 1], fy])
    pot = f.evaluate_to_points(tx, ty, False)
    assert np.all(np.isnan(pot[:4]))
    if kind == "laplace":
        assert not np.any(np.isfinite(pot[4:12]))
    elif kind == "k0":
        assert np.all(pot[4:12] == 0)
    n_pairs = 9 * 40 + 24
    scale = np.abs(ref).max() + np.abs(tau).sum()
    assert np.abs(pot[12:] - ref).max() <= n_pairs * EPS * scale
