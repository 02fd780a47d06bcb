"""The strip moment loop (gqt_strip.cu) against the step loop: several FP64 Chebyshev steps
per launch on plane lattices. The ELL format keeps the step loop, so the same operator in
that format is the reference: every T_k is bit-identical (read through left = a unit
vector, whose moments are single elements of T_k), and the moments are the same
compensated sums in another order."""
from __future__ import annotations

import numpy as np
import pytest

import gpuqt_b200 as g

pytestmark = pytest.mark.gpu

GRAPHENE = [
    [(1, 0, 1), (0, 0, 1), (0, -1, 3)],
    [(0, 0, 0), (-1, 0, 0), (0, 0, 2)],
    [(0, 0, 3), (-1, 0, 3), (0, 0, 1)],
    [(1, 0, 2), (0, 0, 2), (0, 1, 0)],
]
SQUARE = [[(-1, 0, 0), (1, 0, 0), (0, 1, 0), (0, -1, 0)]]
TRIANGLE = [[(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (1, -1, 0), (-1, 1, 0)]]
FAR = [[(1, 0, 0), (-1, 0, 0), (0, 3, 0), (0, -3, 0)]]  # reaches 3 columns


def lattice(hops, n0, n1, *, pbc=(True, True), flux=False, emax=9.3, seed=0):
    """ELL arrays of n0 lines of n1 cells; flux: complex hoppings of period 3 in the line
    number (or, with open boundaries, short rows)."""
    no, z = len(hops), len(hops[0])
    n = n0 * n1 * no
    i = np.arange(n)
    o, c = i % no, i // no
    y, x = c % n1, c // n1
    tab = np.array(hops)[o]
    tx, ty = x[:, None] + tab[..., 0], y[:, None] + tab[..., 1]
    ok = np.ones((n, z), bool)
    if not pbc[0]:
        ok &= (tx >= 0) & (tx < n0)
    if not pbc[1]:
        ok &= (ty >= 0) & (ty < n1)
    nl = ((tx % n0) * n1 + ty % n1) * no + tab[..., 2]
    hr, hi = np.full((n, z), -1.1), np.zeros((n, z))
    if flux:
        ph = 2 * np.pi / 3 * (x % 3)[:, None] * np.sign(tab[..., 1])
        hr, hi = -1.1 * np.cos(ph), -1.1 * np.sin(ph)
    order = np.argsort(~ok, axis=1, kind="stable")
    take = lambda a: np.take_along_axis(a, order, 1)  # noqa: E731
    cnt = ok.sum(1)
    pad = np.arange(z)[None, :] >= cnt[:, None]
    rng = np.random.default_rng(seed)
    return dict(n=n, max_neighbor=z, energy_max=emax, neighbor_number=cnt,
                neighbor_list=np.where(pad, i[:, None], take(nl)).reshape(-1),
                potential=rng.uniform(-1, 1, n), hopping_real=np.where(pad, 0, take(hr)).reshape(-1),
                hopping_imag=np.where(pad, 0, take(hi)).reshape(-1))


CASES = [
    # (hops, lines, cells per line, options): one strip and several, lines shorter than a
    # strip, fewer lines than steps, segments of one line, odd edges, each row length
    (GRAPHENE, 8, 4, {}), (GRAPHENE, 37, 53, {}), (GRAPHENE, 301, 157, {}),
    (SQUARE, 9, 10, {}), (SQUARE, 2, 900, {}), (SQUARE, 17, 24, {}), (SQUARE, 400, 9, {}),
    (SQUARE, 150, 141, {}), (SQUARE, 641, 611, {}), (SQUARE, 331, 20, {"emax": 1e-140}),
    (TRIANGLE, 40, 47, {"pbc": (True, False)}), (FAR, 60, 61, {}),
    (SQUARE, 63, 58, {"flux": True}), (TRIANGLE, 33, 21, {"pbc": (True, False), "flux": True}),
    (SQUARE, 50, 45, {"pbc": (False, True)}), (GRAPHENE, 30, 29, {"pbc": (True, False)}),
    (SQUARE, 31, 64, {"pbc": (False, False), "flux": True}),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_strip_loop_equals_step_loop(case):
    hops, n0, n1, opt = CASES[case]
    opt = dict(opt)
    scale = opt.get("emax", 0.0) == 1e-140  # the division's long form: scaled potentials
    ell = lattice(hops, n0, n1, **opt)
    if scale:
        for k in ("potential", "hopping_real", "hopping_imag"):
            ell[k] = ell[k] * 1e-141
    H = g.Hamiltonian(**ell)
    assert H.format == g.FORMAT_CODED
    n = ell["n"]
    rng = np.random.default_rng(case)
    ph = rng.uniform(0, 2 * np.pi, n)
    phi = g.Vector.from_host(np.cos(ph), np.sin(ph))
    left = g.Vector.from_host(np.sin(3 * ph), np.cos(5 * ph))
    M = 23
    g.reset_launch_count()
    direct = g.moments(H, left, phi, M)
    launches = g.launch_count()
    sym = g.moments_doubled(H, phi, M) if not opt.get("flux") else None
    sites = sorted({0, 1, n1 - 1, n - 1, n // 2, n // 3, *rng.integers(0, n, 5).tolist()})
    units = []
    for s in sites:
        e = np.zeros(n)
        e[s] = 1.0
        units.append(g.Vector.from_host(e, np.zeros(n)))
    elements = [g.moments(H, e, phi, M) for e in units]
    H.set_format(g.FORMAT_ELL)
    g.reset_launch_count()
    want = g.moments(H, left, phi, M)
    assert launches < g.launch_count(), "the strip loop runs in fewer launches"
    # compensated sums: a few ulp of the sum of absolute products, at most n per moment
    np.testing.assert_allclose(direct[0], want[0], rtol=0, atol=1e-15 * n)
    np.testing.assert_allclose(direct[1], want[1], rtol=0, atol=1e-15 * n)
    if sym is not None:
        ws = g.moments_doubled(H, phi, M)
        np.testing.assert_allclose(sym[0], ws[0], rtol=0, atol=1e-15 * n)
    for e, got in zip(units, elements):
        w = g.moments(H, e, phi, M)
        assert np.array_equal(got[0], w[0]) and np.array_equal(got[1], w[1])


def test_strip_loop_does_not_depend_on_the_set_length():
    """A short set is the prefix of a long one, bit for bit, wherever its last launch ends."""
    H = g.Hamiltonian(**lattice(SQUARE, 64, 81))
    ph = np.random.default_rng(1).uniform(0, 2 * np.pi, H.n)
    phi = g.Vector.from_host(np.cos(ph), np.sin(ph))
    long = g.moments(H, phi, phi, 60)
    for M in range(1, 17):
        got = g.moments(H, phi, phi, M)
        assert np.array_equal(got[0], long[0][:M]) and np.array_equal(got[1], long[1][:M])


def slab(n0, n1, n2):
    """Cubic n0 x n1 x n2, periodic: lines of n1 * n2 sites, a reach of n2 columns."""
    n = n0 * n1 * n2
    i = np.arange(n)
    z, y, x = i % n2, i // n2 % n1, i // (n1 * n2)
    at = lambda a, b, c: ((a % n0) * n1 + b % n1) * n2 + c % n2  # noqa: E731
    nl = np.stack([at(x + 1, y, z), at(x - 1, y, z), at(x, y + 1, z), at(x, y - 1, z),
                   at(x, y, z + 1), at(x, y, z - 1)], 1)
    return dict(n=n, max_neighbor=6, energy_max=9.0, neighbor_number=np.full(n, 6),
                neighbor_list=nl.reshape(-1), potential=np.cos(1.7 * i),
                hopping_real=np.full(6 * n, -1.0), hopping_imag=np.zeros(6 * n))


ROUTES = [
    # the operator; whether the direct and the symmetric loop run in strips
    (lambda: lattice(SQUARE, 250, 260), True, True),
    (lambda: lattice(SQUARE, 6500, 10), False, False),      # 10 of a strip's 64 columns
    (lambda: lattice(GRAPHENE, 7000, 3), False, False),
    (lambda: lattice(FAR, 60, 61), True, True),
    (lambda: slab(64, 65, 2), True, True),
    (lambda: slab(64, 64, 6), False, False),                # half of the columns are halo
    (lambda: lattice(SQUARE, 500, 500, flux=False, pbc=(False, True)), True, True),
    (lambda: lattice(GRAPHENE, 300, 300, flux=True), False, False),  # complex, rows of three
    (lambda: lattice(SQUARE, 99, 90, flux=True), True, True),
]


@pytest.mark.parametrize("case", range(len(ROUTES)))
def test_strips_only_where_they_are_faster(case):
    make, direct, sym = ROUTES[case]
    ell = make()
    H = g.Hamiltonian(**ell)
    assert H.format == g.FORMAT_CODED
    n, M = ell["n"], 41
    ph = np.random.default_rng(case).uniform(0, 2 * np.pi, n)
    phi = g.Vector.from_host(np.cos(ph), np.sin(ph))
    calls = (lambda: g.moments(H, phi, phi, M), lambda: g.moments_doubled(H, phi, M))

    def run(call):
        g.reset_launch_count()
        mu = call()
        return mu[0] + 1j * mu[1], g.launch_count()

    got = [run(c) for c in calls]
    H.set_format(g.FORMAT_ELL)
    for (mu, launches), strips, call in zip(got, (direct, sym), calls):
        want, steps = run(call)
        assert (launches < steps) == strips and (strips or launches == steps)
        np.testing.assert_allclose(mu, want, rtol=0, atol=1e-15 * n)


# rows of six with a Hermitian flux along the lines (doubled hops across them: a reach of 1)
SIX = [[(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 1, 0), (0, -1, 0)]]
ROWS = [(hops, n0, n1, pbc, flux)
        for hops, n0, n1 in ((GRAPHENE, 30, 29), (SQUARE, 48, 61), (SIX, 36, 45))
        for pbc in ((True, True), (True, False)) for flux in (False, True)]


@pytest.mark.parametrize("case", range(len(ROWS)))
def test_every_kind_of_row_in_both_loops(case):
    """Rows of 3, 4 and 6, full and short, real and complex, direct and symmetric: the 24
    kernels."""
    hops, n0, n1, pbc, flux = ROWS[case]
    ell = lattice(hops, n0, n1, pbc=pbc, flux=flux, emax=9.9)
    H = g.Hamiltonian(**ell)
    n, M = ell["n"], 40
    ph = np.random.default_rng(case).uniform(0, 2 * np.pi, n)
    phi = g.Vector.from_host(np.cos(ph), np.sin(ph))
    left = g.Vector.from_host(np.sin(3 * ph), np.cos(5 * ph))
    e = np.zeros(n)
    e[n // 2 + 1] = 1.0
    unit = g.Vector.from_host(e, np.zeros(n))
    calls = (lambda: g.moments(H, left, phi, M), lambda: g.moments_doubled(H, phi, M),
             lambda: g.moments(H, unit, phi, M))

    def run(call):
        g.reset_launch_count()
        mu = call()
        return mu[0] + 1j * mu[1], g.launch_count()

    strips = [run(c) for c in calls]
    H.set_format(g.FORMAT_ELL)
    steps = [run(c) for c in calls]
    for (mu, launches), (want, count) in zip(strips, steps):
        assert launches < count
        np.testing.assert_allclose(mu, want, rtol=0, atol=1e-15 * n)
    assert np.array_equal(strips[2][0], steps[2][0])  # elements of T_k, bit for bit


def test_the_largest_shape_element_by_element():
    """Above 1.4 million sites a launch takes 3 steps of 128 columns: elements of T_k at a
    strip's and a segment's edges, odd numbers of lines and columns."""
    n0, n1 = 1201, 1203
    ell = lattice(SQUARE, n0, n1)
    H = g.Hamiltonian(**ell)
    n, M = ell["n"], 20
    ph = np.random.default_rng(0).uniform(0, 2 * np.pi, n)
    phi = g.Vector.from_host(np.cos(ph), np.sin(ph))
    sites = [0, n - 1, n1 - 1, n // 2, *(k * n1 + j for k in (56, 57, 58, 600)
                                         for j in (110, 120, 121, 241))]
    units = []
    for s in sites:
        e = np.zeros(n)
        e[s] = 1.0
        units.append(g.Vector.from_host(e, np.zeros(n)))
    g.reset_launch_count()
    got = [g.moments(H, e, phi, M) for e in units]
    launches = g.launch_count()
    H.set_format(g.FORMAT_ELL)
    g.reset_launch_count()
    want = [g.moments(H, e, phi, M) for e in units]
    assert launches < g.launch_count()
    for a, w in zip(got, want):
        assert np.array_equal(a[0], w[0]) and np.array_equal(a[1], w[1])


def test_lattices_of_several_shapes_side_by_side():
    """Lattices whose launches take different amounts of shared memory share a kernel: replayed
    in turn, and captured at the same time by threads, each gives its own moments."""
    import threading

    def model(k, n0, n1):
        H = g.Hamiltonian(**lattice(SQUARE, n0, n1, seed=k))
        ph = np.random.default_rng(k).uniform(0, 2 * np.pi, H.n)
        return H, g.Vector.from_host(np.cos(ph), np.sin(ph))

    sizes = ((40, 44), (250, 260), (640, 700))  # 6 steps of 32 and of 64 columns, 4 of 96
    models = [model(k, *s) for k, s in enumerate(sizes)]
    lengths = range(20, 60)
    want = [[g.moments(H, x, x, M) for M in lengths] for H, x in models]
    for M in (20, 33):
        for _ in range(2):
            for (H, x), w in zip(models, want):
                got = g.moments(H, x, x, M)
                assert np.array_equal(got[0], w[M - 20][0])
                assert np.array_equal(got[1], w[M - 20][1])
    bad = []

    def work(k):
        try:
            for _ in range(2):
                H, x = model(k, *sizes[k])  # nothing captured yet
                for M, w in zip(lengths, want[k]):
                    got = g.moments(H, x, x, M)
                    if not (np.array_equal(got[0], w[0]) and np.array_equal(got[1], w[1])):
                        bad.append((k, M))
                H.close()
        except Exception as e:  # reported by the assertion below
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]
