"""The FP64 pair loops at the edges of their tiles and series.

A point set of at most Ncutoff points is one leaf, whose evaluation is the
direct sum, so the pair loop stands alone: it is compared with a direct sum in
extended precision (Laplace) or scipy's Bessel functions.  Bound: each kernel
value is within a few ulp, each of n additions rounds once, so the error is at
most (n + 16) eps sum_j (|G_ij| + 1) |tau_j| (+ 1: the logarithm is accurate to
2^-53 absolutely where it is small).
"""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]

EPS = 2.0 ** -52


def cloud(n, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.standard_normal(n)


def direct(kind, k, x, y, tau):
    """(sum, sum of magnitudes) with pairs of equal coordinates left out"""
    from scipy import special
    ld = np.longdouble
    dx, dy = x[:, None].astype(ld) - x[None, :], y[:, None].astype(ld) - y[None, :]
    r2 = dx * dx + dy * dy
    same = r2 == 0
    r2[same] = 1
    if kind == "laplace":
        g = -np.log(r2) / (4 * ld(np.pi))
    else:
        g = special.k0(float(k) * np.sqrt(r2).astype(float)).astype(ld) / (2 * ld(np.pi))
    g[same] = 0
    return (g @ tau.astype(ld)).astype(float), ((np.abs(g) + 1) @ np.abs(tau)).astype(float)


def fmm(kind, k, x, y, cutoff, **kw):
    import pykifmm2d_b200 as P
    kern = P.LaplaceKernel() if kind == "laplace" else P.ModifiedHelmholtzKernel(k)
    f = P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), 24, cutoff, **kw)
    f.build_tree()
    f.precompute()
    return f


# wavenumbers on either side of each series length (t = (k r)^2 up to 8 k^2 W^2,
# W = 2), and where most pairs are beyond the series
KERNELS = [("laplace", 0.0), ("k0", 0.04), ("k0", 0.17), ("k0", 0.34), ("k0", 3.0), ("k0", 60.0)]


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 17, 22, 32, 33, 63, 64, 65, 200])
@pytest.mark.parametrize("kind,k", KERNELS)
def test_one_leaf_is_the_direct_sum(kind, k, n):
    x, y, tau = cloud(n, n)
    if n > 8:
        x[5], y[5] = x[2], y[2]  # an exact duplicate
    for cutoff in (n, 300):
        f = fmm(kind, k, x, y, cutoff)
        assert f.tree_info().levels == 1
        f.build_expansions(tau)
        ref, mag = direct(kind, k, x, y, tau)
        for _ in range(2):  # a second evaluation on the same expansions
            pot = f.evaluate_to_points(x, y, True)
            assert np.all(np.abs(pot - ref) <= (n + 16) * EPS * mag)


@pytest.mark.parametrize("kind,k", KERNELS[:2])
def test_self_pairs_are_infinite_without_check_self(kind, k):
    x, y, tau = cloud(40, 3)
    f = fmm(kind, k, x, y, 64)
    f.build_expansions(np.abs(tau))
    assert np.all(np.isposinf(f.evaluate_to_points(x, y, False)))


@pytest.mark.parametrize("n,cutoff", [(300, 3), (900, 9), (2500, 31), (2500, 33), (6000, 150)])
@pytest.mark.parametrize("kind,k", [("laplace", 0.0), ("k0", 0.3), ("k0", 12.0)])
def test_leaf_tiles_vs_oracle(kind, k, n, cutoff):
    from oracle import oracle as O
    x, y, tau = cloud(n, 7)
    f = fmm(kind, k, x, y, cutoff)
    f.build_expansions(tau)
    pot = f.evaluate_to_points(x, y, True)
    o = O.OracleFMM(x, y, 0 if kind == "laplace" else 1, k, 24, cutoff)
    o.build_expansions(tau)
    ref = o.evaluate_to_points(x, y, True)
    assert np.abs(pot - ref).max() / np.abs(ref).max() <= 1e-9  # the bound of the plain form's other tests


def direct_complex(kind, k, x, y, tau):
    from scipy import special
    dx, dy = x[:, None] - x[None, :], y[:, None] - y[None, :]
    r = np.sqrt(dx * dx + dy * dy)
    same = r == 0
    r[same] = 1
    if kind == "h0":
        g = 0.25j * special.hankel1(0, k * r)
    elif kind == "k0":
        g = special.k0(k * r) / (2 * np.pi) + 0j
    else:
        g = -np.log(r) / (2 * np.pi) + 0j
    g[same] = 0
    return g @ tau, (np.abs(g) + 1) @ np.abs(tau)


@pytest.mark.parametrize("n", [1, 2, 9, 22, 32, 33, 64, 65, 130])
@pytest.mark.parametrize("kind,k", [("h0", 0.04), ("h0", 0.17), ("h0", 0.34), ("h0", 4.0), ("h0", 40.0),
                                    ("laplace", 0.0), ("k0", 0.2), ("k0", 9.0)])
def test_one_leaf_complex(kind, k, n):
    """The complex pair loops; scipy's Bessel functions are good to about 1e-15
    of the function's size near its zeros, hence 64 eps per term."""
    import pykifmm2d_b200 as P
    x, y, tau = cloud(n, n)
    tau = tau + 1j * np.random.default_rng(n + 1).standard_normal(n)
    if n > 8:
        x[5], y[5] = x[2], y[2]
    kern = {"h0": P.HelmholtzKernel, "k0": P.ModifiedHelmholtzKernel}.get(kind, lambda k: P.LaplaceKernel())(k)
    f = P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), 24, 200, True)
    f.build_tree()
    f.precompute()
    f.build_expansions(tau)
    ref, mag = direct_complex(kind, k, x, y, tau)
    pot = f.evaluate_to_points(x, y, True)
    assert np.all(np.abs(pot - ref) <= (n + 64) * EPS * mag)


@pytest.mark.parametrize("nequiv", [4, 6, 8, 10, 12, 16, 18, 20, 24, 28, 30, 32])
@pytest.mark.parametrize("n,cutoff", [(700, 20), (9000, 9), (60000, 9)])
def test_fp64_m2l_shapes(n, cutoff, nequiv):
    """Every number of row tiles, row and column padding, column runs and both
    tile sizes of the FP64 M2L: the complex form works on states of 2 Nequiv, the
    real one of Nequiv, and with a real kernel they are the same sums.  Their
    check-to-equivalent inverses are eliminated differently, so the results
    differ by rounding times the condition of E2C, about Nequiv / 2 (r2 /
    r1)^(Nequiv / 2), over at most eight levels."""
    import pykifmm2d_b200 as P
    x, y, tau = cloud(n, 11)
    kern = P.LaplaceKernel()
    pots = []
    for cplx in (False, True):
        f = P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), nequiv, cutoff, cplx)
        f.build_tree()
        f.precompute()
        f.build_expansions(tau + 0j if cplx else tau)
        pots.append(f.evaluate_to_points(x, y, True))
    r21 = (4 - np.sqrt(2) - 0.02) / (np.sqrt(2) + 0.01)
    tol = 8 * EPS * nequiv / 2 * r21 ** (nequiv / 2)
    assert np.abs(pots[1].imag).max() <= tol * np.abs(pots[0]).max()
    assert np.abs(pots[1].real - pots[0]).max() <= tol * np.abs(pots[0]).max()


def direct_targets(kind, k, x, y, tau, tx, ty):
    """(sum over sources not at the target, sum of magnitudes, sum of |tau| / distance)"""
    from scipy import special
    ld = np.longdouble
    dx, dy = tx[:, None].astype(ld) - x[None, :], ty[:, None].astype(ld) - y[None, :]
    r2 = dx * dx + dy * dy
    same = r2 == 0
    r2[same] = 1
    r = np.sqrt(r2)
    if kind == "laplace":
        g = -np.log(r2) / (4 * ld(np.pi)) + 0j
    elif kind == "k0":
        g = special.k0(k * r.astype(float)) / (2 * np.pi) + 0j
    else:
        g = 0.25j * special.hankel1(0, k * r.astype(float))
    g[same] = 0
    inv = np.where(same, 0, np.abs(tau)[None, :] / r).sum(1)
    return (g @ tau).astype(complex), ((np.abs(g) + 1) @ np.abs(tau)).astype(float), inv.astype(float)


@pytest.mark.parametrize("m", [1, 31, 32, 33, 63, 64, 65, 129, 2049, 5000])
@pytest.mark.parametrize("kind,k,precision", [("laplace", 0.0, "fp64"), ("laplace", 0.0, "mixed"), ("k0", 0.3, "fp64"),
                                              ("k0", 2.0, "mixed"), ("h0", 1.0, "fp64")])
def test_targets_of_one_leaf(kind, k, precision, m):
    """Item sizes of the target groups, targets on sources, and targets outside
    the root box.  FP64 bound as above.  Mixed: offsets are rounded to 2^-24 of the
    box width W = 8 (targets outside it lie within W), which moves a kernel value
    by that over the distance, and FP32 sums of n terms round n times."""
    import pykifmm2d_b200 as P
    n, w = 50, 8.0
    x, y, tau = cloud(n, 5)
    rng = np.random.default_rng(m)
    tx, ty = rng.uniform(-1.5, 1.5, m), rng.uniform(-1.5, 1.5, m)
    tx[:3], ty[:3] = x[:3][:m], y[:3][:m]
    kern = {"h0": P.HelmholtzKernel, "k0": P.ModifiedHelmholtzKernel}.get(kind, lambda k: P.LaplaceKernel())(k)
    f = P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), 24, 64, kind == "h0",
              precision=precision)
    f.build_tree()
    f.precompute()
    f.build_expansions(tau)
    ref, mag, inv = direct_targets(kind, k, x, y, tau, tx, ty)
    pot = f.evaluate_to_points(tx, ty, True)
    tol = (n + 64) * EPS * mag
    if precision == "mixed":
        tol = 2.0 ** -23 * ((n + 16) * mag + w * inv)
    assert np.all(np.abs(pot - ref) <= tol)


@pytest.mark.parametrize("kind,k,cplx", [("laplace", 0.0, False), ("k0", 5.0, False), ("h0", 3.0, True)])
def test_targets_at_the_sources_fp64(kind, k, cplx):
    """Separate targets that are the source points (reordered) give the values at
    the sources: the same sums in another order."""
    import pykifmm2d_b200 as P
    n = 20000
    x, y, tau = cloud(n, 9)
    x[:5000] *= 0.01
    y[:5000] *= 0.01
    kern = {"h0": P.HelmholtzKernel, "k0": P.ModifiedHelmholtzKernel}.get(kind, lambda k: P.LaplaceKernel())(k)
    f = P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), 24, 40, cplx)
    f.build_tree()
    f.precompute()
    f.build_expansions(tau)
    at = f.evaluate_to_points(x, y, True)
    p = np.random.default_rng(1).permutation(n)
    pot = f.evaluate_to_points(x[p].copy(), y[p].copy(), True)
    _, mag, _ = direct_targets(kind, k, x, y, tau, x[:64], y[:64])
    assert np.abs(pot - at[p]).max() <= n * EPS * mag.max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_expansions_of_a_rebuilt_tree(precision):
    """The expansions are cleared once per tree: an object whose points move to
    other trees (more and fewer nodes, empty leaves in other places), with
    several applies on each, gives what a new object gives."""
    import pykifmm2d_b200 as P
    kern = P.LaplaceKernel()
    make = lambda x, y: P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), 24, 20,
                              precision=precision)
    x, y, tau = cloud(6000, 2)
    f = make(x, y)
    for seed, squeeze in ((2, 1.0), (3, 0.02), (4, 1.0), (5, 0.3)):
        nx, ny, _ = cloud(6000, seed)
        nx[:4000] *= squeeze
        x[:], y[:] = nx, ny
        f.build_tree()
        f.precompute()
        for t in (tau * 3, tau):
            f.build_expansions(t)
            pot = f.evaluate_to_points(x, y, True).copy()
        g = make(x.copy(), y.copy())
        g.build_expansions(tau)
        np.testing.assert_array_equal(pot, g.evaluate_to_points(g.x, g.y, True))


@pytest.mark.parametrize("n", [1, 2, 7, 22, 31, 33, 63, 64, 65, 130, 200])
@pytest.mark.parametrize("k", [0.3, 2.0, 12.0])
def test_one_leaf_k0_mixed(k, n):
    """The FP32 near pass alone, with pairs on both sides of k r = 2 (where the
    packed series ends).  Bound with u = 2^-23: a block adds at most 32 values,
    a value is within 16 u (|G| + 1), and coordinates rounded relative to the box
    move r by at most 2 u, the value by 2 u / (2 pi r) < u / r."""
    x, y, tau = cloud(n, 100 + n)
    if n > 8:
        x[5], y[5] = x[2], y[2]
    f = fmm("k0", k, x, y, 300, precision="mixed")
    assert f.tree_info().levels == 1
    f.build_expansions(tau)
    pot = f.evaluate_to_points(x, y, True)
    ref, mag = direct("k0", k, x, y, tau)
    r = np.hypot(x[:, None] - x[None, :], y[:, None] - y[None, :])
    r[r == 0] = 1
    assert np.all(np.abs(pot - ref) <= 50 * 2.0 ** -23 * (mag + (1 / r) @ np.abs(tau)))


@pytest.mark.parametrize("n,cutoff", [(1, 5), (2, 5), (33, 64), (300, 300), (511, 512), (2000, 700), (1500, 1025)])
@pytest.mark.parametrize("kind,k", [("laplace", 0.0), ("k0", 3.0)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_planned_near_field(precision, kind, k, n, cutoff):
    """Trees of one or two levels have no far field: the planned apply is the near
    matrices alone, with rows on both sides of the staged charges' length.  FP32
    rows: charge and matrix value rounded once each, at most 65 products a lane."""
    x, y, tau = cloud(n, n + 1)
    f = fmm(kind, k, x, y, cutoff, precision=precision, planned=True)
    assert f.tree_info().levels <= 2
    f.build_expansions(tau)
    ref, mag = direct(kind, k, x, y, tau)
    bound = (n + 16) * EPS * mag if precision == "fp64" else 70 * 2.0 ** -23 * mag
    for _ in range(2):
        assert np.all(np.abs(f.evaluate_to_points(x, y, True) - ref) <= bound)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,cutoff", [(900, 9), (90000, 20)])
def test_planned_near_field_under_way(precision, n, cutoff):
    """The planned near pass starts with the apply: evaluations that use it, that do
    not (self pairs kept, or other targets), and applies never evaluated."""
    x, y, tau = cloud(n, 5)
    f = fmm("laplace", 0.0, x, y, cutoff, precision=precision, planned=True)
    f.build_expansions(tau)
    a = f.evaluate_to_points(x, y, True)
    f.build_expansions(-tau)
    f.build_expansions(tau)
    other = f.evaluate_to_points(x[:50] + 1e-3, y[:50], False)
    self_pairs = f.evaluate_to_points(x, y, False)
    assert np.all(np.isfinite(other)) and (precision == "mixed" or np.all(np.isinf(self_pairs)))
    b = f.evaluate_to_points(x, y, True)
    f.build_expansions(tau)
    np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(a, f.evaluate_to_points(x, y, True))


@pytest.mark.parametrize("n,cutoff", [(900, 9), (90000, 20)])
@pytest.mark.parametrize("precision,planned", [("fp64", True), ("mixed", True), ("mixed", False)])
def test_evaluation_in_a_callers_capture(precision, planned, n, cutoff):
    """A capture that the caller begins after the apply holds the evaluation alone: it
    cannot wait for a near pass that is under way, and replays on later densities."""
    import torch
    x, y, tau = (torch.as_tensor(v, device="cuda") for v in cloud(n, 8))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    f = fmm("laplace", 0.0, x, y, cutoff, precision=precision, planned=planned, stream=stream.cuda_stream)
    pot, ref = torch.zeros_like(tau), torch.zeros_like(tau)
    f.build_expansions(tau)
    f.evaluate_to_points(x, y, True, out=ref)
    f.synchronize()
    f.build_expansions(tau)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        f.evaluate_to_points(x, y, True, out=pot)
    with torch.cuda.stream(stream):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(pot, ref)
    f.build_expansions(tau.flip(0).contiguous())
    f.evaluate_to_points(x, y, True, out=ref)
    with torch.cuda.stream(stream):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(pot, ref)
