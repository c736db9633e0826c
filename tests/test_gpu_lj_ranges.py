"""Lennard-Jones evaluators at the ends of their ranges: coordinates in large
units, sums of many comparable terms, energies of very unequal pairs, cutoffs
seen from far out, coordinates that are not finite.
"""
import numpy as np
import pytest

from minim_gb300 import abi, runtime
from oracle.oracle import Oracle
from tests.workloads import Rng

pytestmark = pytest.mark.gpu


def _grid(n, seed=3):
    """n points of a cubic grid of spacing 1.08 with noise of 0.05."""
    k = int(np.ceil(n ** (1.0 / 3)))
    idx = np.indices((k,) * 3).reshape(3, -1).T[:n].astype(float)
    return 1.08 * idx + 0.1 * (Rng(seed).uniform(3 * n).reshape(n, 3) - 0.5)


@pytest.mark.parametrize("n", [33, 65, 80, 96, 130, 300])
def test_padding_is_out_of_reach(n):
    """A cluster with sigma = 1e5 around (1e6 (n + 1), 0, 0): no padding particle
    of a tile may stand near it.  A coordinate split into two FP32 parts is good
    to 2^-48 of 3e8, 1.1e-11 sigma, and the energy's and the force's relative
    derivatives are below 20 / sigma: 2e-9 with the sums' own error."""
    sigma = 1e5
    p = abi.lj(sigma=sigma)
    x = (sigma * (_grid(n) - 2.0) + np.array([1e6 * (n + 1), 0.0, 0.0])).ravel()
    eo, go = Oracle(p, x).energy_gradient()
    gmax = np.max(np.abs(go))
    inst = runtime.Instance(p, x)
    e, g = inst.energy_gradient(x)
    assert abs(e - eo) <= 2e-9 * abs(eo) and np.max(np.abs(g - go)) <= 2e-9 * gmax
    e, g = inst.eval_kernel(abi.EVAL_FP64S_CTA, x)
    assert abs(e - eo) <= 2e-9 * abs(eo) and np.max(np.abs(g - go)) <= 2e-7 * gmax


def _crystal(n, seed):
    """A cut of n particles of a face-centred cubic crystal near its minimum, with noise of 0.03."""
    a = 2 ** (1 / 6) * np.sqrt(2) * 0.985
    k = int(np.ceil((n / 4) ** (1 / 3))) + 1
    r = np.arange(-k, k + 1, dtype=float)
    c = np.stack(np.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 1, 3)
    pts = (c + np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]])).reshape(-1, 3) * a
    pts = pts[np.argsort(np.sum((pts - 0.1 * a) ** 2, axis=1), kind="stable")[:n]]
    return pts + 0.03 * Rng(seed).normal(3 * n).reshape(n, 3)


@pytest.mark.parametrize("n", [38, 300, 1000, 1024])
def test_force_sums(n):
    """The FP64 gradient's error against 64 bits in units of the root of the sum
    of its squared terms.  A term is good to some 2^-43.5 (eight roundings of
    2^-47 and the coordinates' split, times up to 14) and the sums have to add
    less than that: 1.2e-13 rms with every sum normalised term by term, on a
    CPU; a low part that gathers 500 terms' roundings makes it 2.0e-13."""
    sq, cnt = 0.0, 0
    for seed in range(3):
        pts = _crystal(n, 100 * n + seed)
        g = runtime.Instance(abi.lj(), pts.ravel()).gradient().reshape(n, 3)
        for i in range(0, n, 200):
            d = pts[i:i + 200, None, :].astype(np.longdouble) - pts[None].astype(np.longdouble)
            r2 = (d * d).sum(2)
            own = np.arange(len(d))
            r2[own, i + own] = 1
            iv = 1 / r2
            iv[own, i + own] = 0
            l6 = iv ** 3
            t = -24 * d * ((2 * l6 * l6 - l6) * iv)[..., None]
            q = (g[i:i + 200] - t.sum(1)) / np.sqrt((t * t).sum(1))
            sq += float((q * q).sum())
            cnt += q.size
    assert np.sqrt(sq / cnt) <= 1.5e-13


@pytest.mark.parametrize("n", [13, 55, 64, 96])
def test_energy_sums(n):
    """The FP64 energy's relative error against 64 bits over 200 crystals, rms.
    Normalised sums, term by term, leave 2.5e-15, 1.4e-15, 1.3e-15 and 1.1e-15
    at these sizes; a tenth more for the 200."""
    sq = 0.0
    for seed in range(200):
        pts = _crystal(n, 1000 * n + seed)
        d = pts[:, None, :].astype(np.longdouble) - pts[None].astype(np.longdouble)
        i6 = (d * d).sum(2)[np.triu_indices(n, 1)] ** -3
        eo = 4 * (i6 * i6 - i6).sum()
        inst = runtime.Instance(abi.lj(), pts.ravel())
        e, _ = inst.energy_gradient(pts.ravel())
        sq += float(((e - eo) / eo) ** 2)
    assert np.sqrt(sq / 200) <= 1.1 * {13: 2.5e-15, 55: 1.4e-15, 64: 1.3e-15, 96: 1.1e-15}[n]


def test_fp32_energy_keeps_small_terms():
    """150 sites 1000 apart, each a pair of particles a quarter apart (energy 4 x
    16773120, exact in FP32 as is each of its steps) among twelve neighbours of
    some -0.1 each.  Every pair's own error is at most 1e-6 of |r^-12| + |r^-6|, in
    all below 15 of each a site; a sum that rounds at 1 loses tenths a site."""
    ring = np.array([[a, b, 0] for a in (-1, 1) for b in (-1, 1)] + [[a, 0, b] for a in (-1, 1) for b in (-1, 1)]
                    + [[0, a, b] for a in (-1, 1) for b in (-1, 1)], float)
    site = np.concatenate([[[0, 0, 0], [0.25, 0, 0]], ring])
    pts = np.concatenate([site + [1000.0 * k, 0, 0] for k in range(150)])
    pts = pts[np.argsort(Rng(8).uniform(len(pts)), kind="stable")]
    d = site[:, None] - site[None]
    r2 = (d * d).sum(2)[np.triu_indices(len(site), 1)]
    assert np.sum(r2 ** -6 + r2 ** -3) - (16.0 ** 6 + 16.0 ** 3) < 15
    exact = 150 * 4 * np.sum(r2 ** -6 - r2 ** -3)
    inst = runtime.Instance(abi.lj(), pts.ravel())
    # (sites see one another at 1000 apart: 4e-18 a pair)
    for gradient in (True, False):
        e, _ = inst.eval_kernel(abi.EVAL_FP32_GRID, pts.ravel(), gradient=gradient)
        assert abs(e - exact) <= 150 * 4 * 15 * 1e-6, e - exact
    # single minimisations' own evaluations, on one CTA and on a cluster (coordinates fixed: the first energy is the last)
    for sites in (3, 6, 20):
        some = np.concatenate([site + [1000.0 * k, 0, 0] for k in range(sites)])
        some = some[np.argsort(Rng(sites).uniform(len(some)), kind="stable")]
        inst = runtime.Instance(abi.lj(), some.ravel(), fixed=list(range(some.size)))
        r = inst.minimise(abi.minimiser("lbfgs", tol=1e-9, max_iter=5, precision="fp32"))
        assert abs(r.energy - exact * sites / 150) <= sites * 4 * 15 * 1e-6, (sites, r.energy)


@pytest.mark.parametrize("n", [13, 40, 64, 90, 200, 256, 400])
def test_cta_evaluation_is_the_batch_kernels(n):
    """The stage evaluations on one CTA run the pair code of a batched L-BFGS
    run: the energies of a run that cannot move (every coordinate fixed) agree
    but for the order of a few FP64 additions."""
    x = _grid(n, seed=n).ravel().astype(np.float32).astype(np.float64)
    for precision, path in (("fp32", abi.EVAL_FP32_CTA), ("mixed", abi.EVAL_FP64S_CTA)):
        inst = runtime.Instance(abi.lj(), x, fixed=list(range(3 * n)))
        b = runtime.Batch()
        b.add(inst, abi.minimiser("lbfgs", tol=1e-9, max_iter=5, precision=precision))
        r = b.run(64 if n <= 96 else (128 if n <= 192 else 256))[0]
        assert precision == "fp32" or r.fp64_iters > 0
        e, _ = inst.eval_kernel(path, x)
        assert abs(e - r.energy) <= 4e-15 * abs(e), (precision, e, r.energy)


def test_cutoff_from_far_out():
    """Pairs a millionth inside and outside the cutoff, 1e8 from the origin: the
    pairs counted are those of the FP64 criterion.  (Coordinates are good to
    2^-48 of 1e8 there, 4e-7: an energy of -0.0163 a pair to 4e-8.)"""
    for n in (32, 300, 2100):
        m = n // 2
        pts = np.zeros((2 * m, 3))
        pts[0::2, 0] = pts[1::2, 0] = 1e8 + 16.0 * np.arange(m)
        pts[1::2, 0] += 2.5 + np.where(np.arange(m) % 2 == 0, -1e-6, 1e-6)
        p = abi.lj(cutoff=2.5)
        inst, o = runtime.Instance(p, pts.ravel()), Oracle(p, pts.ravel())
        eo = o.energy()
        assert abs(eo + 0.0163169 * ((m + 1) // 2)) < 1e-5 * m
        e, _ = inst.energy_gradient(pts.ravel())
        assert abs(e - eo) <= 4e-7 * m
        assert abs(inst.energy(pts.ravel()) - eo) <= 4e-7 * m


@pytest.mark.parametrize("n", [13, 40, 80, 300, 2100])
@pytest.mark.parametrize("cutoff", [0.0, 2.5])
def test_not_finite(n, cutoff):
    """A NaN coordinate makes the energy NaN, and its particle's force; without a
    cutoff everyone's.  A particle at infinity is outside every cutoff."""
    p = abi.lj(cutoff=cutoff)
    x = _grid(n)
    bad = x.copy()
    bad[n // 2, 1] = np.nan
    inst = runtime.Instance(p, x.ravel())
    e, g = inst.energy_gradient(bad.ravel())
    assert np.isnan(e) and np.isnan(inst.energy(bad.ravel()))
    g = g.reshape(n, 3)
    assert np.isnan(g[n // 2, 1])
    if cutoff == 0:
        assert np.all(np.isnan(g[:, 1]))
        return
    away = np.sum((np.delete(x, n // 2, 0) - x[n // 2]) ** 2, axis=1) > 9
    assert np.all(np.isfinite(np.delete(g, n // 2, 0)[away]))
    far = x.copy()
    far[n // 2, 1] = np.inf
    rest = np.delete(x, n // 2, 0)
    eo, go = Oracle(p, rest.ravel()).energy_gradient()
    e, g = inst.energy_gradient(far.ravel())
    assert abs(e - eo) <= 1e-12 * abs(eo) and abs(inst.energy(far.ravel()) - eo) <= 1e-12 * abs(eo)
    others = np.delete(g.reshape(n, 3), n // 2, 0)
    assert np.max(np.abs(others.ravel() - go)) <= 1e-12 * n * np.max(np.abs(go))


@pytest.mark.parametrize("spacing", [1.08, 2.4])
@pytest.mark.parametrize("n,ctas", [(511, 1), (512, 1), (513, 1), (700, 1), (1023, 8), (1024, 8), (1025, 8), (1100, 2),
                                    (2047, 0), (2048, 0), (2049, 0)])
def test_cutoff_rows_and_cells(n, ctas, spacing):
    """On either side of where rows end and the cell list begins, one CTA, cluster
    and grid: the energy of a run that cannot move is the oracle's, dense and
    dilute."""
    p = abi.lj(cutoff=2.5)
    x = (_grid(n) * (spacing / 1.08)).ravel().astype(np.float32).astype(np.float64)
    eo = Oracle(p, x).energy()
    inst = runtime.Instance(p, x, fixed=list(range(3 * n)))
    for precision, tol in (("fp32", 2e-6), ("fp64", 1e-12)):
        mp = abi.minimiser("lbfgs", tol=1e-9, max_iter=5, precision=precision)
        if ctas:
            b = runtime.Batch()
            b.add(inst, mp)
            r = b.run(256, ctas)[0]
        else:
            r = inst.minimise(mp)
        assert abs(r.energy - eo) <= tol * abs(eo)


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("x", [0.3, np.nan, np.inf, -np.inf, 1e200, 1e30])
def test_single_particle(x, ndim):
    """One particle has no pair: no energy and no force wherever it is."""
    pos = np.array([0.5, x, -0.2])[:ndim]
    inst = runtime.Instance(abi.lj(ndim=ndim), pos)
    e, g = inst.energy_gradient(pos)
    assert e == 0 and np.all(g == 0) and inst.energy(pos) == 0
    for precision in ("fp32", "mixed", "fp64"):
        for method in (dict(method="lbfgs"), dict(method="fire", dt_max=0.02)):
            inst.coords = pos
            r = inst.minimise(abi.minimiser(max_iter=5, tol=1e-6, precision=precision, **method))
            assert r.status == abi.RES_CONVERGED and r.energy == 0


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("unit", [1e6, 1e15])
def test_particle_far_along_an_axis(unit, axis):
    """A particle far out along one coordinate meets nothing, no padding either
    (which stood at (1e6 k, 0, 0)): the others' energy and forces are theirs alone."""
    n = 80
    p = abi.lj()
    x = _grid(n, seed=6)
    x[n - 1] = 0.0
    eo, go = Oracle(p, x[:n - 1].ravel()).energy_gradient()
    inst = runtime.Instance(p, x.ravel())
    for k in range(n, 98):
        x[n - 1, axis] = k * unit
        tol = 1e-12 + (n * (5.0 / unit) ** 6 if unit < 1e10 else 0.0)
        e, g = inst.energy_gradient(x.ravel())
        assert abs(e - eo) <= tol * abs(eo) and np.max(np.abs(g[:-3] - go)) <= 1e-12 * n * np.max(np.abs(go))
        for path, ge, ee in ((abi.EVAL_FP32_CTA, 1e-5, 2e-6), (abi.EVAL_FP64S_CTA, 2e-7, 1e-12)):
            xs = x.astype(np.float32).astype(np.float64) if path == abi.EVAL_FP32_CTA else x
            es, gs = Oracle(p, xs[:n - 1].ravel()).energy_gradient()
            e, g = inst.eval_kernel(path, xs.ravel())
            assert abs(e - es) <= ee * abs(es) and np.max(np.abs(g[:-3] - gs)) <= ge * np.max(np.abs(gs)), (k, path)
