"""The work a user has this library do, as cases that can be timed and compared.

A case is one call, or one correlation step, of a linear-scaling transport run on a
tight-binding model: a set of KPM moments (DOS, VAC), the VAC step around it, or the
Bessel-series time evolution of an MSD step. The models are the lattices of the
workloads module (square, graphene in its 4-orbital cell, cubic, a batch of square
lattices) and graphene with vacancies (the reference's review example), with Anderson
disorder, in the sizes users run: a few hundred sites while a model is set up, 65,536
sites and odd sizes for ordinary runs, millions for converged ones.

kind       square | graphene | cubic | vacancy | batch
n0 n1 n2   lattice cells (batch: models' edge lengths are drawn between n0 and n1)
form       fp64 | fp32 | fp32r: the arithmetic form of the moment recurrence
op         dos     moments of a random-phase state with itself (left = right)
           dos_sym the same set from half the steps (moments_doubled)
           vac     one VAC correlation step: the current operator, a moment set with
                   left != right, and the evolution of both states
           evolve  the time evolutions of one MSD step: [X, U(dt)] on one state, U(dt)
                   on another
nvec       random vectors per launch
moments    Chebyshev moments (vac: of its set); dt: time step times E_max
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gpuqt_b200 as g

FORMS = {"fp64": g.FP64, "fp32": g.FP32, "fp32r": g.FP32R}
SQUARE = [[(-1, 0, 0, 0), (1, 0, 0, 0), (0, 1, 0, 0), (0, -1, 0, 0)]]
CUBIC = [[(1, 0, 0, 0), (-1, 0, 0, 0), (0, 1, 0, 0), (0, -1, 0, 0), (0, 0, 1, 0), (0, 0, -1, 0)]]
GRAPHENE = [
    [(1, 0, 0, 1), (0, 0, 0, 1), (0, -1, 0, 3)],
    [(0, 0, 0, 0), (-1, 0, 0, 0), (0, 0, 0, 2)],
    [(0, 0, 0, 3), (-1, 0, 0, 3), (0, 0, 0, 1)],
    [(1, 0, 0, 2), (0, 0, 0, 2), (0, 1, 0, 0)],
]
# hops, orbital x positions, cell length along x, hopping, Anderson width, E_max
LATTICES = {
    "square": (SQUARE, [0.0], 1.0, -1.0, 2.0, 5.0),
    "graphene": (GRAPHENE, [0.866, 0.0, 0.0, 0.866], 1.7321, -2.7, 1.0, 8.7),
    "vacancy": (GRAPHENE, [0.866, 0.0, 0.0, 0.866], 1.7321, -2.7, 0.0, 8.7),
    "cubic": (CUBIC, [0.0], 1.0, -1.0, 16.5, 15.0),
}
VACANCIES = 0.01  # 200,000 of 20 million sites in the reference's review example


def listed():
    return [
        # setting a model up: a few hundred sites, a short set; latency is all there is
        dict(name="square_tiny_dos", kind="square", n0=17, n1=24, n2=1, form="fp64", op="dos",
             nvec=1, moments=200, dt=0.0),
        # the 256 x 256 square lattice of the published FP64 configuration: a VAC step
        dict(name="square_256_vac", kind="square", n0=256, n1=256, n2=1, form="fp64", op="vac",
             nvec=1, moments=1000, dt=5.0),
        # an ordinary size with odd edges, one DOS set
        dict(name="graphene_odd_dos", kind="graphene", n0=301, n1=157, n2=1, form="fp64",
             op="dos", nvec=1, moments=600, dt=0.0),
        # the graphene configuration (2,097,152 sites), part of its 3000 moments
        dict(name="graphene_2m_dos", kind="graphene", n0=1024, n1=512, n2=1, form="fp64",
             op="dos", nvec=1, moments=1000, dt=0.0),
        # the same model in the precision form, 16 random vectors per launch
        dict(name="graphene_2m_fp32", kind="graphene", n0=1024, n1=512, n2=1, form="fp32",
             op="dos", nvec=16, moments=150, dt=0.0),
        # the fastest route to a symmetric set: FP32 recurrence from half the steps
        dict(name="graphene_1m_fp32r_sym", kind="graphene", n0=640, n1=409, n2=1, form="fp32r",
             op="dos_sym", nvec=16, moments=400, dt=0.0),
        # symmetric set in FP64 (para.in kpm_doubling)
        dict(name="square_1m_sym", kind="square", n0=1000, n1=1001, n2=1, form="fp64",
             op="dos_sym", nvec=1, moments=1000, dt=0.0),
        # the 3D Anderson model at its transition (256^3 in the published configuration)
        dict(name="cubic_2m_dos", kind="cubic", n0=128, n1=128, n2=128, form="fp64", op="dos",
             nvec=1, moments=400, dt=0.0),
        # the same model with 16 batched vectors, direct set
        dict(name="cubic_90_fp32r", kind="cubic", n0=90, n1=91, n2=88, form="fp32r", op="dos",
             nvec=16, moments=200, dt=0.0),
        # graphene with vacancies: ragged rows on the ELL arrays
        dict(name="vacancy_1m_dos", kind="vacancy", n0=512, n1=500, n2=1, form="fp64", op="dos",
             nvec=1, moments=500, dt=0.0),
        # disorder realisations of uneven sizes in one launch, 32 vectors each
        dict(name="batch_fp32", kind="batch", n0=64, n1=700, n2=8, form="fp32", op="dos",
             nvec=32, moments=100, dt=0.0),
        # the evolutions of one MSD step of 1 fs
        dict(name="graphene_1m_evolve", kind="graphene", n0=512, n1=511, n2=1, form="fp64",
             op="evolve", nvec=1, moments=0, dt=13.2),
    ]


def draw(rng):
    """One more call of the same ranges: sizes log-uniform, odd edges included, its work
    bounded by the listed cases'."""
    kind = rng.choice(["square", "square", "graphene", "graphene", "cubic", "vacancy", "batch"])
    if kind == "batch":
        return dict(kind=kind, n0=rng.randint(20, 90), n1=rng.randint(150, 600),
                    n2=rng.randint(2, 9), form=rng.choice(["fp32", "fp32r"]),
                    op=rng.choice(["dos", "dos_sym"]), nvec=16, moments=2 * rng.randint(20, 60),
                    dt=0.0)
    form = rng.choice(["fp64", "fp64", "fp64", "fp32", "fp32r"])
    nvec = {"fp64": rng.choice([1, 1, 1, 4]), "fp32": rng.choice([1, 16]), "fp32r": 16}[form]
    op = rng.choice(["dos", "dos", "dos_sym", "vac", "evolve"])
    if form != "fp64" and op in ("vac", "evolve"):
        op = "dos"
    # sites times vectors: 300 to 2 million (16 million for many vectors)
    total = math.exp(rng.uniform(math.log(300.0), math.log(2.0e6)))
    if nvec == 16:
        total = math.exp(rng.uniform(math.log(16 * 300.0), math.log(1.6e7)))
    sites = total / nvec
    per_cell = 4 if kind in ("graphene", "vacancy") else 1
    cells = max(sites / per_cell, 16.0)
    if kind == "cubic":
        e = cells ** (1.0 / 3.0)
        n0, n1 = (max(4, round(e * rng.uniform(0.7, 1.4))) for _ in range(2))
        n2 = max(4, round(cells / (n0 * n1)))
    else:
        n0 = max(4, round(math.sqrt(cells) * math.exp(rng.uniform(-0.7, 0.7))))
        n1, n2 = max(4, round(cells / n0)), 1
    n = n0 * n1 * n2 * per_cell * nvec
    # moments log-uniform in 100 .. 2000, fewer where a step is long
    m = math.exp(rng.uniform(math.log(100.0), math.log(2000.0)))
    m = int(max(40.0, min(m, (1.2e9 if nvec < 16 else 3.0e9) / n)))
    return dict(kind=kind, n0=n0, n1=n1, n2=n2, form=form, op=op, nvec=nvec,
                moments=0 if op == "evolve" else m,
                dt=round(rng.uniform(1.0, 15.0), 3) if op in ("vac", "evolve") else 0.0)


# ------------------------------------------------------------------ models and states
def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + salt)


def _lattice(kind, n0, n1, n2, seed, width=None, salt=0):
    """ELL arrays [n, z] (CUDA tensors): rows in the reference's site order, x slowest."""
    hops, pos, ax, t, w, emax = LATTICES[kind]
    if width is not None:
        w, emax = width, 4.0 + width / 2 + 0.1
    dev = "cuda"
    no, z = len(hops), len(hops[0])
    n = n0 * n1 * n2 * no
    i = torch.arange(n, device=dev)
    o, c = i % no, i // no
    cz, cy, cx = c % n2, (c // n2) % n1, c // (n1 * n2)
    tab = torch.tensor(hops, device=dev)  # [no, z, 4]
    dx = torch.tensor([[h[0] * ax + pos[h[3]] - pos[k] for h in hops[k]] for k in range(no)],
                      dtype=torch.float64, device=dev)
    d = tab[o]
    nl = ((((cx[:, None] + d[..., 0]) % n0) * n1 + (cy[:, None] + d[..., 1]) % n1) * n2
          + (cz[:, None] + d[..., 2]) % n2) * no + d[..., 3]
    xx = dx[o]
    gen = _generator(seed, 1 + 16 * salt)
    pot = (torch.rand(n, generator=gen, device=dev, dtype=torch.float64) - 0.5) * w
    hop = torch.full((n, z), t, dtype=torch.float64, device=dev)
    cnt = torch.full((n,), z, dtype=torch.int64, device=dev)
    if kind == "vacancy":
        keep = torch.rand(n, generator=gen, device=dev) >= VACANCIES
        new = torch.cumsum(keep, 0) - 1
        ok = keep[nl][keep]
        order = torch.sort((~ok).to(torch.int8), dim=1, stable=True).indices
        nl = torch.gather(new[nl][keep], 1, order)
        xx = torch.gather(xx[keep], 1, order)
        cnt = ok.sum(1)
        pad = torch.arange(z, device=dev)[None, :] >= cnt[:, None]
        n = int(keep.sum())
        nl = torch.where(pad, torch.arange(n, device=dev)[:, None], nl)
        hop, xx, pot = hop[keep].masked_fill(pad, 0.0), xx.masked_fill(pad, 0.0), pot[keep]
    return dict(n=n, z=z, emax=emax, cnt=cnt, nl=nl, hop=hop, xx=xx, pot=pot)


def _models(case, seed):
    if case["kind"] != "batch":
        return [_lattice(case["kind"], case["n0"], case["n1"], case["n2"], seed)]
    # n2 square lattices, edges log-uniform in [n0, n1], Anderson widths in [0.5, 4]: the
    # sizes belong to the case, the disorder to the seed
    rs = np.random.RandomState(11)
    edge = np.exp(rs.uniform(math.log(case["n0"]), math.log(case["n1"]), case["n2"]))
    width = rs.uniform(0.5, 4.0, case["n2"])
    return [_lattice("square", int(round(e)), int(round(e)), 1, seed, float(w), k)
            for k, (e, w) in enumerate(zip(edge, width))]


def _sites(case):
    per = 4 if case["kind"] in ("graphene", "vacancy") else 1
    if case["kind"] != "batch":
        return case["n0"] * case["n1"] * case["n2"] * per
    rs = np.random.RandomState(11)
    edge = np.exp(rs.uniform(math.log(case["n0"]), math.log(case["n1"]), case["n2"]))
    return int(sum(round(e) ** 2 for e in edge))


def _phases(case, model, seed, salt):
    """Random-phase vectors [nvec, n], exact in the storage form of the case."""
    gen = _generator(seed, 2 + 16 * salt)
    a = torch.rand(case["nvec"], model["n"], generator=gen, device="cuda", dtype=torch.float64)
    a = a * (2.0 * math.pi)
    re, im = torch.cos(a), torch.sin(a)
    if case["form"] != "fp64":
        re, im = re.float().double(), im.float().double()
    return re, im


def _ell(m):
    f = lambda t: t.cpu().numpy().reshape(-1)  # noqa: E731
    return dict(n=m["n"], max_neighbor=m["z"], energy_max=m["emax"],
                neighbor_number=f(m["cnt"].int()), neighbor_list=f(m["nl"].int()),
                potential=f(m["pot"]), hopping_real=f(m["hop"]),
                hopping_imag=np.zeros(m["n"] * m["z"]), xx=f(m["xx"]))


class _Device:
    """A Vector's device data for torch.as_tensor (FP64: [n, nvec] complex). The tensor
    keeps this object, and with it the Vector, alive."""

    def __init__(self, v):
        self.vector = v
        self.__cuda_array_interface__ = dict(shape=(v.n, v.nvec), typestr="<c16", version=3,
                                             data=(v.data_ptr, False))


def prepare(case, seed):
    models = _models(case, seed)
    phases = [_phases(case, m, seed, k) for k, m in enumerate(models)]
    store = g.FP64 if case["form"] == "fp64" else g.FP32
    if case["kind"] == "batch":
        H = g.Hamiltonian.batch([_ell(m) for m in models])
        re, im = H.scatter([(a.cpu().numpy(), b.cpu().numpy()) for a, b in phases])
    else:
        H = g.Hamiltonian(**_ell(models[0]))
        re, im = (a.cpu().numpy() for a in phases[0])
    phi = g.Vector.from_host(re, im, nvec=case["nvec"], precision=store)
    s = dict(case=case, H=H, phi=phi)
    if case["op"] in ("vac", "evolve"):
        # the work vectors the correlation stages keep
        s.update(a=g.Vector(phi.n, phi.nvec), b=g.Vector(phi.n, phi.nvec),
                 c=g.Vector(phi.n, phi.nvec))
        for k in "abc":
            s["t" + k] = torch.as_tensor(_Device(s[k]), device="cuda")
    return s


def run(s):
    case, H, phi = s["case"], s["H"], s["phi"]
    if case["op"] == "dos":
        re, im = g.moments(H, phi, phi, case["moments"], precision=FORMS[case["form"]])
        return re + 1j * im
    if case["op"] == "dos_sym":
        re, im = g.moments_doubled(H, phi, case["moments"], precision=FORMS[case["form"]])
        return re + 1j * im
    if case["op"] == "vac":
        # one step of the VAC stage: a = left state, b = right state, c = V left
        s["a"].copy_from(phi)
        g.apply_current(H, s["a"], s["b"])
        g.apply_current(H, s["a"], s["c"])
        re, im = g.moments(H, s["b"], s["c"], case["moments"], precision=FORMS[case["form"]])
        g.evolve(H, -1, case["dt"], s["a"])
        g.evolve(H, -1, case["dt"], s["b"])
        return dict(mu=re + 1j * im, left=s["ta"], right=s["tb"])
    # the evolutions of an MSD step: [X, U] of the state, U on both states, their sum
    s["a"].copy_from(phi)
    s["b"].copy_from(phi)
    g.evolvex(H, 1, case["dt"], s["b"])
    g.evolve(H, 1, case["dt"], s["a"])
    s["c"].copy_from(s["b"])
    s["c"].add(s["a"])
    return dict(state=s["ta"], state_x=s["tb"], total=s["tc"])


def _bessel(x):
    """J_0(x) .. J_m(x), up to the first m >= 2 with |J_m| < 1e-15 (Miller's downward
    recurrence, normalised by J_0 + 2 (J_2 + J_4 + ...) = 1)."""
    top = int(x) + 60
    top += top % 2
    j = np.zeros(top + 2)
    j[top] = 1e-300
    for m in range(top, 0, -1):
        j[m - 1] = 2.0 * m / x * j[m] - j[m + 1]
        if abs(j[m - 1]) > 1e200:
            j[m - 1:] *= 1e-200
    j /= j[0] + 2.0 * j[2::2].sum()
    last = next(m for m in range(2, top) if abs(j[m]) < 1e-15)
    return j[:last]


def work(case):
    """One pass: the operator (potential, neighbour and hopping of every entry where they
    differ from site to site) and the input vectors read once, the outputs written once;
    the arithmetic of every Chebyshev step."""
    n, v = _sites(case), case["nvec"]
    z = {"square": 4, "batch": 4, "cubic": 6}.get(case["kind"], 3)
    elem = 16 if case["form"] == "fp64" else 8
    entry = 20 * z if case["kind"] == "vacancy" else z
    # potential 2, complex hopping times vector and sum 8 z, scale 2, 2 t - T_{k-2} 2
    apply_flops = 6 + 8 * z
    nbytes = n * (8 + entry) + n * v * elem
    flops = 0
    if case["op"] in ("dos", "vac"):
        flops += case["moments"] * n * v * (apply_flops + 8)
        nbytes += 16 * case["moments"] * v
    if case["op"] == "dos_sym":
        flops += case["moments"] // 2 * n * v * (apply_flops + 12)
        nbytes += 16 * case["moments"] * v
    if case["op"] in ("vac", "evolve"):
        terms = len(_bessel(case["dt"]))
        both = 2 if case["op"] == "vac" else 1 + 2.5  # evolvex: two rows and the commutator
        flops += both * terms * n * v * (apply_flops + 4)
        nbytes += (2 if case["op"] == "vac" else 3) * n * v * elem
    return dict(bytes=float(nbytes), flops=float(flops))


def tolerance(case):
    """About four times what another order of the sums, or of the roundings in FP32, was
    seen to change: FP64 sets and states are within 1e-14 of their values; direct FP32
    sets within 2e-8 (the rounding of each element averages over the sites), symmetric
    ones within 5e-7 (every product of a T_k with itself carries its rounding)."""
    if case["form"] == "fp64":
        return dict(rel=1e-13, max=1e-12)
    if case["op"] == "dos":
        return dict(rel=1e-7, max=2e-6)
    return dict(rel=2e-6, max=2e-5)


# ------------------------------------------------------------------ the same in torch
class _H:
    """The model's operator on [n, nvec] complex128 tensors."""

    def __init__(self, m):
        self.m = m
        self.nl, self.hop = m["nl"], m["hop"]

    def _sum(self, x, w):
        out = None
        for k in range(self.m["z"]):
            t = w[:, k, None] * x[self.nl[:, k]]
            out = t if out is None else out + t
        return out

    def apply(self, x):
        return (self.m["pot"][:, None] * x + self._sum(x, self.hop)) / self.m["emax"]

    def commutator(self, x):
        return -self._sum(x, self.hop * self.m["xx"]) / self.m["emax"]

    def current(self, x):
        return -1j * self._sum(x, self.hop * self.m["xx"])

    def moments(self, left, right, count):
        mu = []
        t0, t1 = right, self.apply(right)
        for k in range(count):
            t = t0 if k == 0 else t1 if k == 1 else 2 * self.apply(t1) - t0
            if k >= 2:
                t0, t1 = t1, t
            mu.append((left.conj() * t).sum(0))
        return torch.stack(mu, 1)  # [nvec, count]

    def evolve(self, x, direction, dt):
        j = _bessel(dt)
        t0, t1 = x, self.apply(x)
        out = j[0] * t0 + 2 * (-1j * direction) * j[1] * t1
        for m in range(2, len(j)):
            t0, t1 = t1, 2 * self.apply(t1) - t0
            out = out + 2 * (-1j * direction) ** m * j[m] * t1
        return out

    def evolvex(self, x, direction, dt):
        """[X, U(dt)] x from the recurrence of [X, T_m]."""
        j = _bessel(dt)
        t0, t1 = x, self.apply(x)
        x0, x1 = torch.zeros_like(x), self.commutator(x)
        # the reference's first term does not depend on the direction
        out = -2j * j[1] * x1
        for m in range(2, len(j)):
            x0, x1 = x1, 2 * (self.apply(x1) + self.commutator(t1)) - x0
            t0, t1 = t1, 2 * self.apply(t1) - t0
            out = out + 2 * (-1j * direction) ** m * j[m] * x1
        return out


def exact(case, seed):
    models = _models(case, seed)
    if case["kind"] == "batch":
        mus = []
        for k, m in enumerate(models):
            phi = torch.complex(*_phases(case, m, seed, k)).T.contiguous()
            mus.append(_H(m).moments(phi, phi, case["moments"]))
        return torch.stack(mus).cpu().numpy()
    H = _H(models[0])
    phi = torch.complex(*_phases(case, models[0], seed, 0)).T.contiguous()
    if case["op"] in ("dos", "dos_sym"):
        mu = H.moments(phi, phi, case["moments"]).cpu().numpy()
        return mu[0] if case["nvec"] == 1 else mu
    if case["op"] == "vac":
        cur = H.current(phi)
        mu = H.moments(cur, cur, case["moments"]).cpu().numpy()
        return dict(mu=mu[0] if case["nvec"] == 1 else mu, left=H.evolve(phi, -1, case["dt"]),
                    right=H.evolve(cur, -1, case["dt"]))
    a, b = H.evolve(phi, 1, case["dt"]), H.evolvex(phi, 1, case["dt"])
    return dict(state=a, state_x=b, total=a + b)
