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


# (points, Ncutoff): a tree whose near pass starts with the apply, one whose near
# pass starts after the M2M chain, and one with leaves above level 2
TREES = [(900, 9), (90000, 20), (-52, 20)]


def lopsided(n, seed):
    """n < 0: a few points in three quadrants (leaves of level 1), the others in the
    fourth (leaves of level 2, the only ones with a far field)"""
    x, y, tau = cloud(abs(n), seed)
    if n < 0:
        x[12:], y[12:] = np.abs(x[12:]), np.abs(y[12:])
        x[:4], y[:4] = -np.abs(x[:4]), -np.abs(y[:4])
        x[4:8], y[4:8] = -np.abs(x[4:8]), np.abs(y[4:8])
        x[8:12], y[8:12] = np.abs(x[8:12]), -np.abs(y[8:12])
    return x, y, tau


def on_device(*arrays):
    import torch
    return [torch.as_tensor(v, device="cuda") for v in arrays]


@pytest.mark.parametrize("n,cutoff", TREES)
@pytest.mark.parametrize("kind,precision,planned", [("laplace", "mixed", False), ("k0", "mixed", False),
                                                    ("laplace", "fp64", True), ("laplace", "mixed", True)])
def test_replay_after_an_apply_never_evaluated(kind, precision, planned, n, cutoff):
    """The near pass of an apply may still be under way when a graph of the same plan
    is launched; the evaluation that follows is of the graph's densities."""
    import torch
    x, y, tau, other = on_device(*lopsided(n, 8), np.random.default_rng(9).standard_normal(abs(n)))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    f = fmm(kind, 2.0, x, y, cutoff, precision=precision, planned=planned, stream=stream.cuda_stream)
    if n < 0:
        nodes, _ = f.export_tree()
        assert np.any((nodes[:, 0] == 1) & (nodes[:, 3] == 1) & (nodes[:, 6] > 0))
    pot, at = torch.zeros_like(tau), torch.zeros_like(tau)
    f.capture_apply(tau, pot, True)
    f.replay()
    f.synchronize()
    ref = pot.clone()
    elsewhere = x[:5] + 1e-3, y[:5].clone()
    for look in (False, True):
        pot.zero_()
        torch.cuda.synchronize()
        f.build_expansions(other)
        if look:
            f.evaluate_to_points(*elsewhere, False)
        f.replay()
        f.evaluate_to_points(x, y, True, out=at)
        f.synchronize()
        assert torch.equal(pot, ref) and torch.equal(at, ref)


@pytest.mark.parametrize("n,cutoff", TREES)
@pytest.mark.parametrize("kind", ["laplace", "k0"])
def test_batch_after_an_apply_never_evaluated(kind, n, cutoff):
    import torch
    from pykifmm2d_b200.serving import PackedBatch
    x, y, tau, other = on_device(*lopsided(n, 8), np.random.default_rng(9).standard_normal(abs(n)))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    # every plan on the batch's stream, so that only the near passes run beside it
    fs = [fmm(kind, 2.0, x, y, cutoff, precision="mixed", stream=stream.cuda_stream) for _ in range(2)]
    taus, pots = [tau, other.clone()], [torch.zeros_like(tau) for _ in range(2)]
    batch = PackedBatch(fs, taus, pots, stream)
    batch.launch()
    batch.synchronize()
    refs = [p.clone() for p in pots]
    at = torch.zeros_like(tau)
    for p in pots:
        p.zero_()
    torch.cuda.synchronize()
    for f in fs:
        f.build_expansions(other)
    batch.launch()
    fs[0].evaluate_to_points(x, y, True, out=at)
    batch.synchronize()
    fs[0].synchronize()
    assert all(torch.equal(p, r) for p, r in zip(pots, refs)) and torch.equal(at, refs[0])
    batch.close()


@pytest.mark.parametrize("n,cutoff", TREES)
@pytest.mark.parametrize("kind,precision,planned", [("laplace", "mixed", False), ("k0", "mixed", False),
                                                    ("laplace", "fp64", True)])
@pytest.mark.parametrize("whole", [False, True])
def test_callers_graph_after_an_apply_never_evaluated(kind, precision, planned, n, cutoff, whole):
    """A graph of the caller's holding an evaluation, or a whole apply, replayed
    straight after a build_expansions."""
    import torch
    x, y, tau, other = on_device(*lopsided(n, 8), np.random.default_rng(9).standard_normal(abs(n)))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    f = fmm(kind, 2.0, x, y, cutoff, precision=precision, planned=planned, stream=stream.cuda_stream)
    pot, ref = torch.zeros_like(tau), torch.zeros_like(tau)
    f.build_expansions(tau if whole else other)
    f.evaluate_to_points(x, y, True, out=ref)
    f.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        if whole:
            f.build_expansions(tau)
        f.evaluate_to_points(x, y, True, out=pot)
    for _ in range(3):
        f.build_expansions(other)
        with torch.cuda.stream(stream):
            pot.zero_()
            g.replay()
        torch.cuda.synchronize()
        assert torch.equal(pot, ref)


@pytest.mark.parametrize("kind,iscomplex,precision", [("h0", True, "fp64"), ("laplace", True, "fp64"),
                                                      ("laplace", False, "fp64"), ("laplace", False, "mixed")])
def test_device_arrays_of_any_alignment(kind, iscomplex, precision):
    """Densities and potentials one double past a 16-byte boundary, through the C ABI
    (whose arrays are doubles): the values of aligned ones, eagerly and replayed."""
    import torch
    from pykifmm2d_b200 import _lib as B
    x, y, tau = on_device(*cloud(3000, 6))
    width = 2 if iscomplex else 1
    t = torch.stack([tau, tau.flip(0)], 1).reshape(-1) if iscomplex else tau
    stream = torch.cuda.Stream()
    f = fmm(kind, 2.0, x, y, 40, iscomplex, precision=precision, stream=stream.cuda_stream)
    buf = {off: [torch.zeros(3000 * width + 2, dtype=torch.float64, device="cuda") for _ in range(2)] for off in (0, 1)}
    pots = []
    for off, (bt, bp) in buf.items():
        at, ap = bt[off:off + t.numel()], bp[off:off + t.numel()]
        assert ap.data_ptr() % 16 == 8 * off
        at.copy_(t)
        torch.cuda.synchronize()
        lib = B.load()
        B.check(lib.kifmm_build_expansions(f._plan, at.data_ptr(), B.MEM_DEVICE))
        B.check(lib.kifmm_evaluate_to_sources(f._plan, ap.data_ptr(), 1, B.MEM_DEVICE))
        f.synchronize()
        pots.append(ap.clone())
        ap.zero_()
        torch.cuda.synchronize()
        B.check(lib.kifmm_graph_capture(f._plan, at.data_ptr(), ap.data_ptr(), 1))
        B.check(lib.kifmm_graph_launch(f._plan))
        f.synchronize()
        pots.append(ap.clone())
    assert all(torch.equal(p, pots[0]) for p in pots[1:]) and pots[0].abs().max() > 0


@pytest.mark.parametrize("rebuilt", [False, True])
def test_batch_with_managed_memory(rebuilt):
    """A packed batch whose densities and results are managed memory, of plans whose
    earlier applies used device arrays in place."""
    import ctypes

    from cuda.bindings import runtime
    from pykifmm2d_b200 import _lib as B
    import torch
    lib = B.load()
    stream = torch.cuda.Stream()
    sizes = [3000, 5000]
    fs, arrays, refs, managed = [], [], [], []
    for r, n in enumerate(sizes):
        x, y, tau = on_device(*cloud(n, r))
        torch.cuda.synchronize()
        m = n // 2 if rebuilt else n
        f = fmm("laplace", 0.0, x[:m].contiguous(), y[:m].contiguous(), 40, precision="mixed", stream=stream.cuda_stream)
        f.build_expansions(tau[:m].contiguous())
        f.evaluate_to_points(f.x, f.y, True)
        if rebuilt:
            f.x, f.y = x, y
            f.build_tree()
            f.precompute()
        f.synchronize()
        fs.append(f)
        g = fmm("laplace", 0.0, x, y, 40, precision="mixed", stream=stream.cuda_stream)
        g.build_expansions(tau)
        refs.append(g.evaluate_to_points(x, y, True).cpu().numpy())
        g.synchronize()
        pair = []
        for _ in range(2):
            err, p = runtime.cudaMallocManaged(8 * n, runtime.cudaMemAttachGlobal)
            assert int(err) == 0
            managed.append(p)
            pair.append((int(p), np.ctypeslib.as_array((ctypes.c_double * n).from_address(int(p)))))
        pair[0][1][:] = tau.cpu().numpy()
        pair[1][1][:] = 0
        arrays.append(pair)
    ptrs = [(ctypes.c_void_p * 2)(*[a[k][0] for a in arrays]) for k in (0, 1)]
    plans = (ctypes.c_void_p * 2)(*[f._plan.value for f in fs])
    h = ctypes.c_void_p()
    B.check(lib.kifmm_batch_capture(plans, 2, ptrs[0], ptrs[1], 1, ctypes.c_void_p(stream.cuda_stream), ctypes.byref(h)))
    for _ in range(2):
        for a in arrays:
            a[1][1][:] = 0
        B.check(lib.kifmm_batch_launch(h))
        B.check(lib.kifmm_batch_synchronize(h))
        for a, ref in zip(arrays, refs):
            np.testing.assert_array_equal(a[1][1], ref)
    B.check(lib.kifmm_batch_destroy(h))
    for p in managed:
        runtime.cudaFree(p)


@pytest.mark.parametrize("kind,k,iscomplex,precision", [
    ("laplace", 0.0, False, "fp64"), ("laplace", 0.0, True, "fp64"), ("laplace", 0.0, False, "mixed"),
    ("k0", 2.0, False, "fp64"), ("k0", 60.0, False, "fp64"), ("k0", 2.0, False, "mixed"), ("h0", 2.0, True, "fp64")])
@pytest.mark.parametrize("m", [700, 20000, 300000])
def test_equal_calls_at_targets_give_equal_bits(kind, k, iscomplex, precision, m):
    """The order in which targets are grouped by leaf is not fixed; their sums are.
    Leaves with fewer targets than an item holds, a few items each, and many."""
    x, y, tau = cloud(2000, 3)
    f = fmm(kind, k, x, y, 40, iscomplex, precision=precision)
    f.build_expansions(tau + 0j if iscomplex else tau)
    tx, ty, _ = cloud(m, 4)
    ref = f.evaluate_to_points(tx, ty, False)
    for _ in range(4):
        np.testing.assert_array_equal(f.evaluate_to_points(tx, ty, False), ref)


def log_targets():
    """distances r with exact squares: beside 1, and of 26 random bits over 2^-30 .. 2^20"""
    k = np.arange(3, 27)
    beside = np.concatenate([[1.0], 1 + 2.0 ** -k, 1 - 2.0 ** -k])
    rng = np.random.default_rng(2)
    wide = np.ldexp(np.floor(rng.uniform(0.5, 1, 4000) * 2 ** 26) / 2 ** 26, rng.integers(-29, 21, 4000))
    close = 1 + np.floor(rng.uniform(-0.4, 0.4, 4000) * 2 ** 25) / 2 ** 25
    return np.concatenate([beside, wide, close])


@pytest.mark.parametrize("iscomplex", [False, True])
@pytest.mark.parametrize("at_sources", [False, True])
def test_logarithm_is_relatively_accurate(at_sources, iscomplex):
    """One charge at the origin: the potential is the logarithm of r^2 times its
    scale, to its last bits also where it is small, and zero at r = 1.  Bound: 4.0 ulp
    (an ulp is at most 2^-52 of the value) for the logarithm, one for its scale and
    one for the product with it."""
    r = log_targets()
    r2 = r.astype(np.longdouble) ** 2
    ref = np.where(np.abs(r2 - 1) < 0.5, np.log1p(np.maximum(r2, 0.25) - 1), np.log(r2)) / (-16 * np.arctan(np.longdouble(1)))
    if at_sources:
        x = np.concatenate([[0.0], r])
        y = np.zeros_like(x)
        tau = np.zeros_like(x)
        tau[0] = 1
        f = fmm("laplace", 0.0, x, y, len(x), iscomplex)
        f.build_expansions(tau + 0j if iscomplex else tau)
        pot = f.evaluate_to_points(x, y, True)[1:]
    else:
        f = fmm("laplace", 0.0, np.array([0.0, 1.0]), np.array([0.0, 1.0]), 4, iscomplex)
        f.build_expansions(np.array([1.0, 0.0]) + (0j if iscomplex else 0))
        pot = f.evaluate_to_points(r, 0 * r, True)
        np.testing.assert_array_equal(pot, f.evaluate_to_points(0 * r, r, True))
    assert np.all(np.abs(pot - ref.astype(float)) <= 6.0 * EPS * np.abs(ref).astype(float))
    assert r[0] == 1 and pot[0] == 0


def test_trees_of_moving_points_vs_oracle():
    """Two objects whose points move between clouds of other depths (all with points
    on one circle, so that their deep cells lie side by side), built in turn with
    other work under way: the words of an earlier tree that a build finds in its
    buffers are in none of its cells."""
    import pykifmm2d_b200 as P
    from oracle import oracle as O
    n, cutoff = 40000, 12
    clouds, want = [], []
    for seed, sigma in enumerate((1e-1, 1e-3, 1e-2, 3e-4)):
        rng = np.random.default_rng(seed)
        th = rng.uniform(0, 2 * np.pi, n // 2)
        th[:n // 4] *= sigma
        c = rng.uniform(-0.9, 0.9, (2, 8))[:, rng.integers(0, 8, n - n // 2)]
        z = c + sigma * rng.standard_normal(c.shape)
        clouds.append(np.concatenate([[np.cos(th), np.sin(th)], z], 1))
        want.append(O.OracleTree(clouds[-1][0], clouds[-1][1], cutoff).export()[0])
    clouds = [on_device(*c) for c in clouds]
    kern = P.LaplaceKernel()
    fs = []
    for _ in range(2):
        x, y = (v.clone() for v in clouds[0])
        fs.append(P.FMM(x, y, P.Get_Kernel_Functions(kern), P.prepare_numba_functions_on_the_fly(kern), 32, cutoff,
                        precision="mixed"))
    for i in range(200):
        k, f = (i * 7 // 5) % 4, fs[i % 2]
        f.x.copy_(clouds[k][0])
        f.y.copy_(clouds[k][1])
        f.build_tree()
        f.precompute()
        f.build_expansions(f.x)
        f.evaluate_to_points(f.x, f.y, True)
        if i % 23 < 2:
            np.testing.assert_array_equal(f.export_tree()[0], want[k])


@pytest.mark.parametrize("kind", ["k0", "h0"])
@pytest.mark.parametrize("k", [1e-152, 1e-158, 1e-161, 1e-170])
def test_wavenumbers_whose_square_underflows(kind, k):
    """K0(z) and H0(z) of tiny z are -ln(z / 2) - gamma and its like to the last bit;
    one leaf, so the potential is the direct sum: the rounding of n additions of values
    within a few ulp."""
    n = 30
    x, y, tau = cloud(n, 1)
    x, y = 4e6 * x, 4e6 * y  # (k r)^2 is a normal number again for most k here
    f = fmm(kind, k, x, y, 64, kind == "h0")
    f.build_expansions(tau + 0j if kind == "h0" else tau)
    ld = np.longdouble
    r2 = (x[:, None].astype(ld) - x) ** 2 + (y[:, None].astype(ld) - y) ** 2
    off = ~np.eye(n, dtype=bool)
    g = np.zeros((n, n), dtype=np.clongdouble)
    ln = np.log(ld(k)) + np.log(r2[off]) / 2 - np.log(ld(2)) + ld("0.57721566490153286060651209008240243")
    g[off] = -ln / (8 * np.arctan(ld(1))) + (0.25j if kind == "h0" else 0)
    ref, mag = g @ tau, np.abs(g).astype(float) @ np.abs(tau)
    for pot in (f.evaluate_to_points(x, y, True), f.evaluate_to_points(x.copy(), y.copy(), True)):
        assert np.all(np.abs(pot - ref) <= (n + 16) * EPS * mag)


def test_complex_targets_in_runs():
    """More complex targets than one grouping takes (2^27): the same potentials on
    either side of the boundary as in a call of their own, up to the rounding of 50
    additions."""
    import torch
    n, m, cut = 50, (1 << 27) + 700, 1 << 27
    x, y, tau = on_device(*cloud(n, 2))
    f = fmm("laplace", 0.0, x, y, 64, True)
    f.build_expansions(tau + 0j)
    g = torch.Generator(device="cuda").manual_seed(1)
    tx, ty = (torch.rand(m, generator=g, device="cuda", dtype=torch.float64) for _ in range(2))
    pot = f.evaluate_to_points(tx, ty, False)
    for a, b in ((0, 300), (cut - 300, cut + 300), (m - 300, m)):
        ref = f.evaluate_to_points(tx[a:b].contiguous(), ty[a:b].contiguous(), False)
        assert (pot[a:b] - ref).abs().max() <= (n + 16) * EPS * tau.abs().sum()


@pytest.mark.parametrize("nequiv", [4, 7, 8, 9, 16, 17, 24, 25, 32, 33, 40, 41, 48, 49, 56, 57, 64])
def test_planned_p2m_of_every_number_of_check_points(nequiv):
    """Planned expansions, seen at separate targets (which use no planned matrix), are
    those of the kernels: a check potential is the same sum in another order, carried
    by the condition of the check-to-equivalent solve, about Nequiv / 2 (r2 /
    r1)^(Nequiv / 2), over at most eight levels."""
    x, y, tau = cloud(3000, 5)
    tx, ty, _ = cloud(200, 6)
    pots = []
    for planned in (False, True):
        f = fmm("laplace", 0.0, x, y, 30, nequiv=nequiv, planned=planned)
        f.build_expansions(tau)
        pots.append(f.evaluate_to_points(tx, ty, False))
    r21 = (4 - np.sqrt(2) - 0.02) / (np.sqrt(2) + 0.01)
    tol = 8 * EPS * nequiv / 2 * r21 ** (nequiv / 2)
    assert np.abs(pots[1] - pots[0]).max() <= max(tol, 64 * EPS) * np.abs(pots[0]).max()


def test_planned_leaves_beyond_shared_memory():
    """A planned near pass keeps a leaf's sums in shared memory.  For an Ncutoff that
    does not fit, the evaluation at the sources is refused, as it always was; the apply
    and evaluations elsewhere are not, before or after it."""
    from pykifmm2d_b200 import _lib as B
    n, cutoff = 30100, 30000
    x, y, tau = cloud(n, 1)
    x[4:], y[4:] = np.abs(x[4:]), np.abs(y[4:])  # one quadrant splits: three levels
    x[:4], y[:4] = -np.abs(x[:4]), -np.abs(y[:4])
    tx, ty, _ = cloud(200, 2)
    f = fmm("laplace", 0.0, x, y, cutoff, precision="mixed", planned=True)
    g = fmm("laplace", 0.0, x, y, cutoff, precision="mixed")
    assert f.tree_info().levels == 3
    for h in (f, g):
        h.build_expansions(tau)
    ref = g.evaluate_to_points(tx, ty, False)
    scale = np.abs(ref).max()
    assert np.abs(f.evaluate_to_points(tx, ty, False) - ref).max() <= 1e-9 * scale
    with pytest.raises(B.KifmmError):
        f.evaluate_to_points(x, y, True)
    assert np.abs(f.evaluate_to_points(tx, ty, False) - ref).max() <= 1e-9 * scale
