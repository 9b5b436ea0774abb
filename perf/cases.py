"""The workloads this framework is timed on, through its public Python API
(`su2higgs_gb300.gpu`): pools of independent chains, single lattices, chains
whose fields live on the host, multicanonical runs, gradient flow, measurement
and correlators, in both precisions and for every field content.

A case is a dict of plain values; `prepare` makes what a program has in hand
(the lattice or pool with its uploaded fields), `run` is one pass of the work,
`work` the bytes and operations it cannot do without and `exact` the same
values from plain torch in 64 bits.
"""
import math

import numpy as np
import torch

from su2higgs_gb300 import abi, gpu, workloads

FIELDS = gpu.FIELD_NAMES
ENSEMBLE = ",".join(str(s) for s in workloads.ENSEMBLE_SIDES)


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the batched ensemble of the benchmark: 384 adjoint chains, ten sweeps
        # between measurements, launch shapes from the pool's autotuner
        dict(name="ensemble_384", kind="pool", content="adj", precision=32, chains=384, sides=ENSEMBLE, sweeps=10,
             autotune=True),
        # a quarter of it by a program that leaves the sweep mode to the pool
        dict(name="ensemble_96", kind="pool", content="adj", precision=32, chains=96, sides=ENSEMBLE, sweeps=10,
             autotune=False),
        # a finite-size scan on small volumes: many short chains, latency-bound
        dict(name="small_chains", kind="pool", content="adj", precision=32, chains=48, sides="8,10,12,16", sweeps=10,
             autotune=False),
        # multicanonical chains of the SU(2)xU(1)+singlet theory in one pool
        dict(name="muca_pool", kind="muca_pool", content="su2u1s", precision=32, chains=24, sides="16,20,24,32",
             sweeps=4, autotune=False),
        # a batch step on host arrays: upload, sweeps, measurement, download
        dict(name="cycle_64", kind="cycle", content="adj", precision=32, chains=64, sides="8,12,16,24,32", sweeps=10,
             autotune=False),
        # one large lattice, swept between measurements
        dict(name="fund_128", kind="lattice", content="fund", precision=32, Lx=128, Ly=128, Lz=128, sweeps=5),
        # the reference's plain configuration: FP64, measured every sweep
        dict(name="fund_16_f64", kind="lattice", content="fund", precision=64, Lx=16, Ly=16, Lz=16, sweeps=1),
        # a production lattice of the adjoint theory with unequal sides
        dict(name="adj_ragged", kind="lattice", content="adj", precision=32, Lx=36, Ly=28, Lz=50, sweeps=10),
        # a multicanonical run on one lattice, a check after every half-sweep
        dict(name="muca_96", kind="muca", content="su2u1s", precision=32, Lx=96, Ly=96, Lz=96, sweeps=2),
        # update_lattice() of the reference's program on its own host arrays
        dict(name="host_fundadj_f64", kind="host", content="fundadj", precision=64, Lx=24, Ly=24, Lz=24, sweeps=1),
        # gradient flow of a configuration with its measurements
        dict(name="flow_64", kind="flow", content="adj", precision=32, Lx=64, Ly=64, Lz=64, steps=20, interval=5),
        # correlators of a configuration and of its blocked lattices
        dict(name="correl_48", kind="correl", content="adj", precision=32, Lx=48, Ly=48, Lz=48, levels=2),
    ]


def _even(rng, lo, hi):
    """An even side, spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, 2 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2)))


def draw(rng):
    kind = rng.choice(["pool", "pool", "lattice", "lattice", "lattice", "muca_pool", "cycle", "muca", "host", "flow",
                       "correl"])
    c = dict(kind=kind)
    if kind in ("pool", "muca_pool", "cycle"):
        c["content"] = "su2u1s" if kind == "muca_pool" else rng.choice(["adj", "adj", "fund", "su2u1s", "fundadj"])
        c["precision"] = rng.choice([32, 32, 32, 64])
        f64 = c["precision"] == 64
        c["chains"] = round(math.exp(rng.uniform(math.log(4), math.log(32 if f64 else 128))))
        top = _even(rng, 8, 24 if f64 else 40)
        c["sides"] = ",".join(str(s) for s in sorted({_even(rng, 4, top) for _ in range(4)} | {top}))
        c["sweeps"] = 1 if f64 else rng.randint(2, 8)
        c["autotune"] = False
        return c
    c["content"] = {"muca": "su2u1s", "correl": "adj"}.get(kind) or rng.choice(["adj", "fund", "su2u1s", "fundadj",
                                                                                "higgs2", "pure"])
    c["precision"] = rng.choice([32, 32, 64])
    f64 = c["precision"] == 64
    top = {"correl": 48, "host": 48, "flow": 64}.get(kind, 96)
    for d in "xyz":
        c["L" + d] = _even(rng, 6, min(top, 40) if f64 else top)
    if kind == "flow":
        c["steps"], c["interval"] = rng.randint(4, 24), rng.randint(2, 8)
    elif kind == "correl":
        c["levels"] = rng.randint(0, 2)
    else:
        c["sweeps"] = 1 if f64 or kind == "host" else rng.randint(1, 8)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _couplings(case, g):
    """Couplings of one chain: the ensembles' ranges for the adjoint theory,
    the reference configuration's values otherwise."""
    if case["content"] != "adj":
        return {}
    lo, hi = workloads.ENSEMBLE_BETA
    mlo, mhi = workloads.ENSEMBLE_MSQ_ADJ
    u = torch.rand(2, generator=g, dtype=torch.float64)
    return dict(betasu2=lo + (hi - lo) * float(u[0]), msq_triplet=mlo + (mhi - mlo) * float(u[1]),
                b4=workloads.ENSEMBLE_LAMBDA_ADJ)


def _chains(case, seed):
    """[(params, chain seed)] of the case: one lattice, or a pool's chains."""
    g = torch.Generator().manual_seed(seed)
    if "Lx" in case:
        sides = [(case["Lx"], case["Ly"], case["Lz"])]
    else:
        pick = [int(s) for s in case["sides"].split(",")]
        # sides cycle through the list, so that every seed has the same work
        sides = [(pick[k % len(pick)],) * 3 for k in range(case["chains"])]
    return [(abi.make_params(case["content"], L=L, precision=case["precision"], **_couplings(case, g)),
             1000 * seed + 17 * k) for k, L in enumerate(sides)]


def _host_fields(case, params, seed, pinned=False):
    """FP64 host arrays of consecutive chains in layout order, as near to an
    equilibrated configuration as independent sites get: links around unity,
    scalars of the size they have in the runs.  For the FP32 form the values
    are representable in 32 bits.  Returns {field: (sum of V, ...) array}."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    V = sum(p.sites() for p in params)
    p = params[0]

    def normal(n, s):
        return s * torch.randn(V, n, generator=g, device="cuda", dtype=torch.float64)

    link = normal(12, 0.35).view(V, 3, 4)
    link[..., 0] = 1.0
    out = {"link": link / link.norm(dim=2, keepdim=True)}
    if p.content & abi.U1:
        out["u1"] = normal(3, 0.25)
    for h in range(p.nhiggs()):
        out["d%d" % h] = normal(4, 0.35) + 0.1
    if p.content & abi.TRIPLET:
        out["trip"] = normal(3, 0.4) + 0.1
    if p.content & abi.SINGLET:
        out["sing"] = normal(1, 0.4)[:, 0]
    host = {}
    for n, t in out.items():
        t = t.float().double() if p.precision == 32 else t
        h = torch.empty(t.shape, dtype=torch.float64, pin_memory=pinned)
        h.copy_(t)
        host[n] = h.numpy()
    return host


def _split(params, host):
    """Views of each chain's part of the arrays."""
    out, at = [], 0
    for p in params:
        out.append({n: a[at:at + p.sites()] for n, a in host.items()})
        at += p.sites()
    return out


def prepare(case, seed):
    chains = _chains(case, seed)
    params = [p for p, _ in chains]
    host = _host_fields(case, params, seed, pinned=case["kind"] == "cycle")
    if "Lx" in case:
        lat = gpu.Lattice(params[0], seed=chains[0][1])
        lat.upload(**host)
        s = dict(case=case, lat=lat, sweep=0)
        if case["kind"] == "muca":
            s["weight"] = workloads.muca_weight()
            lat.muca_set(s["weight"].struct)
            for parity in (0, 1):
                lat.calc_orderparam(parity)
        if case["kind"] == "host":
            s["fields"] = host
        return s
    pool = gpu.Pool(params[0], sum(gpu.Pool.chain_bytes(p) for p in params), max_chains=len(params))
    slots = [pool.add(p, seed=cs, chain=k) for k, (p, cs) in enumerate(chains)]
    s = dict(case=case, pool=pool, slots=slots)
    pool.upload_many(slots, _split(params, host))
    if case["kind"] == "muca_pool":
        s["weight"] = workloads.muca_weight()
        for slot in slots:
            pool.muca_set(slot, s["weight"].struct)
    if case["autotune"]:
        pool.autotune()
    if case["kind"] == "cycle":
        s["host"], s["fields"] = host, _split(params, host)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("pool", "muca_pool"):
        s["pool"].run(case["sweeps"])
        sums = s["pool"].measure()
        return {"sums": np.stack([sums[slot] for slot in s["slots"]])}
    if kind == "cycle":
        sums = s["pool"].cycle(s["slots"], s["fields"], case["sweeps"])
        return dict(s["host"], sums=sums)
    lat = s["lat"]
    if kind == "flow":
        return {"rows": lat.grad_flow(0.01 * (case["steps"] - 0.5), 0.01, case["interval"])}
    if kind == "correl":
        out = {"level0": lat.measure_correlators()}
        if case["levels"]:
            for k, rows in enumerate(lat.measure_blocked_correlators((1, 1, 1), case["levels"])):
                out["level%d" % (k + 1)] = rows
        return out
    first = s["sweep"]
    s["sweep"] += case["sweeps"]
    if kind == "host":
        lat.update_lattice_host(first, s["fields"])
        return dict(s["fields"])
    lat.run_sweeps(first, case["sweeps"])
    return {"sums": lat.measure()}


# ---------------------------------------------------------------------------
# the least a pass has to move and to compute
# ---------------------------------------------------------------------------
def _reals(p):
    """Reals per site of the field content."""
    return (12 + (3 if p.content & abi.U1 else 0) + 4 * p.nhiggs() + (3 if p.content & abi.TRIPLET else 0) +
            (1 if p.content & abi.SINGLET else 0))


def _sweep_flops(p):
    """Operations per site of one sweep: the staples and matrix products of
    one update of each link and of scalar_sweeps + 1 of each scalar."""
    nh, trip = p.nhiggs(), bool(p.content & abi.TRIPLET)
    link = 8 * 28 + 28 * nh + (90 if trip else 0) + 80
    scalar = nh * (6 * 28 + 100) + (6 * 45 + 100 if trip else 0) + (60 if p.content & abi.SINGLET else 0)
    return 3 * link + (3 * 120 if p.content & abi.U1 else 0) + (p.scalar_sweeps + 1) * scalar


def _measure_flops(p):
    trip = bool(p.content & abi.TRIPLET)
    return 250 + 130 * p.nhiggs() + (900 if trip else 0) + (100 if p.content & abi.U1 else 0)


def work(case):
    params = [p for p, _ in _chains(case, 0)]
    V, p = sum(q.sites() for q in params), params[0]
    size = case["precision"] // 8
    fields = V * _reals(p) * size
    kind = case["kind"]
    if kind == "flow":
        rows = 1 + -(-case["steps"] // case["interval"])
        return {"bytes": fields, "flops": V * (900 * case["steps"] + _measure_flops(p) * rows)}
    if kind == "correl":
        return {"bytes": fields, "flops": V * 1500}
    flops = V * _sweep_flops(p) * case["sweeps"]
    if kind == "host":
        return {"bytes": 2 * V * _reals(p) * 8, "flops": flops}
    if kind == "cycle":
        return {"bytes": 2 * V * _reals(p) * 8, "flops": flops + V * _measure_flops(p)}
    return {"bytes": 2 * fields, "flops": flops + V * _measure_flops(p)}


# ---------------------------------------------------------------------------
# the same values in 64 bits from plain torch.  Fields are lexicographic
# tensors [z, y, x, ...]; quaternions (a, b, c, d) = a + i(b s1 + c s2 + d s3).
# ---------------------------------------------------------------------------
def _order(L):
    """Storage index of every lexicographic site: EVEN sites first, the
    lexicographic order kept inside each parity."""
    x, y, z = (torch.arange(n) for n in L)
    n = x[None, None, :] + L[0] * (y[None, :, None] + L[1] * z[:, None, None])
    par = (x[None, None, :] + y[None, :, None] + z[:, None, None]) % 2
    return (par * (L[0] * L[1] * L[2] // 2) + n // 2).cuda(), par.cuda()


def _up(f, d, n=1):
    """The field at x + n e_d."""
    return torch.roll(f, -n, dims=2 - d)


def _mul(x, y):
    a, b, c, d = x.unbind(-1)
    e, f, g, h = y.unbind(-1)
    return torch.stack([a * e - b * f - c * g - d * h, a * f + e * b + d * g - c * h,
                        a * g + e * c + b * h - d * f, a * h + e * d + c * f - b * g], -1)


def _dag(x):
    return x * torch.tensor([1.0, -1.0, -1.0, -1.0], dtype=x.dtype, device=x.device)


def _rot(u, t):
    return _mul(_mul(u, torch.nn.functional.pad(t, (1, 0))), _dag(u))[..., 1:]


def _phase(a):
    o = torch.zeros_like(a)
    return torch.stack([torch.cos(a), o, o, -torch.sin(a)], -1)


class _Lattice64:
    """The formulas of the measurements and updates on lexicographic tensors."""

    def __init__(self, p, host):
        self.p = p
        self.idx, self.par = _order(p.L[:3])
        f = {n: torch.from_numpy(np.ascontiguousarray(a)).cuda()[self.idx] for n, a in host.items()}
        self.U = [f["link"][..., d, :] for d in range(3)]
        self.A = [f["u1"][..., d] for d in range(3)] if "u1" in f else None
        self.phi = [f[n] for n in ("d0", "d1") if n in f]
        self.T, self.S = f.get("trip"), f.get("sing")

    def stored(self):
        """The fields as host arrays in storage order."""
        flat = self.idx.reshape(-1)

        def put(t):
            t = t.reshape((flat.numel(),) + t.shape[3:])
            out = torch.empty_like(t)
            out[flat] = t
            return out.cpu().numpy()

        out = {"link": put(torch.stack(self.U, 3))}
        out.update({"d%d" % h: put(f) for h, f in enumerate(self.phi)})
        if self.T is not None:
            out["trip"] = put(self.T)
        return out

    def staple(self, mu):
        """The Wilson staple of U_mu."""
        U, tot = self.U, 0.0
        for nu in range(3):
            if nu != mu:
                tot = tot + _mul(_mul(_up(U[nu], mu), _dag(_up(U[mu], nu))), _dag(U[nu]))
                lo = _mul(_mul(_dag(_up(U[nu], mu)), _dag(U[mu])), U[nu])
                tot = tot + _up(lo, nu, -1)
        return tot

    def scalar_staple(self, f, forward):
        """-sum over directions of the neighbours, transported to the site."""
        s = 0.0
        for d in range(3):
            s = s - forward(d, self.U[d], _up(f, d)) - _up(forward(d, _dag(self.U[d]), f, True), d, -1)
        return s

    def doublet_staple(self, h):
        def hop(d, u, f, back=False):
            w = _mul(u, f)
            return w if self.A is None else _mul(w, _phase(-self.A[d] if back else self.A[d]))
        return self.scalar_staple(self.phi[h], hop)

    def triplet_staple(self):
        return self.scalar_staple(self.T, lambda d, u, t, back=False: _rot(u, t))

    def alpha(self, d1, d2):
        """The plaquette angle of the U(1) the triplet leaves unbroken: the
        argument of tr of the four links projected by (1 + n.sigma)/2."""
        n = self.T / self.T.norm(dim=-1, keepdim=True)
        one = torch.eye(2, dtype=torch.complex128, device=n.device)
        sig = torch.tensor([[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]], dtype=torch.complex128,
                           device=n.device)
        proj = 0.5 * (one + torch.einsum("...k,kij->...ij", n.to(torch.complex128), sig))
        basis = torch.cat([one[None], 1j * sig])
        P = {}
        for d in (d1, d2):
            u = torch.einsum("...k,kij->...ij", self.U[d].to(torch.complex128), basis)
            P[d] = proj @ u @ _up(proj, d)
        m = P[d1] @ _up(P[d2], d1) @ _up(P[d1], d2).mH @ P[d2].mH
        return torch.angle(m.diagonal(dim1=-2, dim2=-1).sum(-1)) * math.sqrt(self.p.betasu2)

    def measure(self):
        p, U, m = self.p, self.U, np.zeros(abi.NMEAS)
        act = 0.0
        wil = 0.0
        for i, j in ((0, 1), (0, 2), (1, 2)):
            plaq = _mul(_mul(U[i], _up(U[j], i)), _dag(_mul(U[j], _up(U[i], j))))
            wil = wil + p.betasu2 * (1.0 - plaq[..., 0])
        m[abi.M_WILSON] = wil.sum()
        act = act + wil
        if self.A is not None:
            u1 = 0.0
            for i, j in ((0, 1), (0, 2), (1, 2)):
                ang = self.A[i] + _up(self.A[j], i) - _up(self.A[i], j) - self.A[j]
                u1 = u1 + p.betau1 * (1.0 - torch.cos(p.r_u1 * ang))
            m[abi.M_U1WILSON] = u1.sum()
            act = act + u1
        mod = [0.5 * f.square().sum(-1) for f in self.phi]
        for h, f in enumerate(self.phi):
            cov = 0.0
            for d in range(3):
                w = _mul(U[d], _up(f, d))
                if self.A is not None:
                    w = _mul(w, _phase(self.A[d]))
                cov = cov + 2.0 * mod[h] - (f * w).sum(-1)
            act = act + cov
            m[abi.M_COV_PHI + 3 * h], m[abi.M_PHI2 + 3 * h], m[abi.M_PHI4 + 3 * h] = (
                cov.sum(), mod[h].sum(), mod[h].square().sum())
        if self.phi:
            act = act + p.msq_phi * mod[0] + p.lambda_phi * mod[0] ** 2
        if len(self.phi) == 2:
            a, b = self.phi
            re = 0.5 * (a * b).sum(-1)
            im = 0.5 * (a[..., 3] * b[..., 0] + a[..., 2] * b[..., 1] - a[..., 1] * b[..., 2] - a[..., 0] * b[..., 3])
            m[abi.M_PHI12_RE], m[abi.M_PHI12_IM] = re.sum(), im.sum()
            f11, f22 = mod
            act = act + (p.msq_phi2 * f22 + p.m12sq_re * re - p.m12sq_im * im + p.lam2 * f22 ** 2 +
                         p.lam3 * f11 * f22 + p.lam4 * (re ** 2 + im ** 2) + p.lam5_re * (re ** 2 - im ** 2) -
                         2 * p.lam5_im * re * im + f11 * (p.lam6_re * re - p.lam6_im * im) +
                         f22 * (p.lam7_re * re + p.lam7_im * im))
        if self.T is not None:
            t2 = 0.5 * self.T.square().sum(-1)
            hop = 0.0
            for d in range(3):
                hop = hop - (self.T * _rot(U[d], _up(self.T, d))).sum(-1)
            act = act + 6.0 * t2 + hop + p.msq_triplet * t2 + p.b4 * t2 ** 2
            m[abi.M_HOP_SIGMA], m[abi.M_SIGMA2], m[abi.M_SIGMA4] = hop.sum(), t2.sum(), t2.square().sum()
            if self.phi:
                act = act + p.a2 * mod[0] * t2
                m[abi.M_PHI2SIGMA2] = (mod[0] * t2).sum()
            q = 0.0
            for (i, j), d, sign in (((1, 2), 0, 1), ((0, 2), 1, -1), ((0, 1), 2, 1)):
                B = sign * self.alpha(i, j)
                q = q + _up(B, d) - B
            m[abi.M_MAGCHARGE], m[abi.M_MAGCHARGE_ABS] = q.sum(), q.abs().sum()
        if self.S is not None:
            S = self.S
            cov = 0.0
            for d in range(3):
                cov = cov + S * S - S * _up(S, d)
            act = act + cov + p.b1_s * S + 0.5 * p.msq_s * S ** 2 + p.b3_s / 3 * S ** 3 + 0.25 * p.b4_s * S ** 4
            m[abi.M_S_COV] = cov.sum()
            for k in range(4):
                m[abi.M_S1 + k] = (S ** (k + 1)).sum()
            if len(self.phi) == 1:
                act = act + 0.5 * p.a1_s * S * mod[0] + 0.5 * p.a2_s * S ** 2 * mod[0]
                m[abi.M_SPHI2], m[abi.M_S2PHI2] = (mod[0] * S).sum(), (mod[0] * S ** 2).sum()
        m[abi.M_ACTION] = act.sum()
        return m

    # -- gradient flow ------------------------------------------------------
    def tree_mass(self):
        """The triplet's mass without its counterterm, which the flow drops."""
        p = self.p
        sigma, zeta, delta, rho = 3.17591153625, 0.08849, 1.942130, -0.313964
        k1, k2, k3, k4 = 0.958382, 0.25 * sigma ** 2 - 0.5 * delta - 0.25, 0.751498, 1.204295
        g2, b4 = 4.0 / p.betasu2, p.b4
        ct = -(4.0 * g2 + 5.0 * b4) * sigma / (4.0 * math.pi)
        ct -= 1.0 / (16.0 * math.pi ** 2) * (
            (20.0 * b4 * g2 - 10.0 * b4 ** 2) * (math.log(6.0 / g2) + zeta) +
            20.0 * b4 * g2 * (0.25 * sigma ** 2 - delta) +
            2.0 * g2 ** 2 * (1.25 * sigma ** 2 + math.pi / 3.0 * sigma - 6.0 * delta - 6.0 * rho + 4.0 * k1 - k2 - k3 -
                             3.0 * k4))
        return p.msq_triplet - ct

    def flow_step(self, dt):
        p, U = self.p, self.U
        new = []
        for mu in range(3):
            s = self.staple(mu) * (-p.betasu2 / 8.0)
            if self.T is not None:
                pad = torch.nn.functional.pad
                s = s + _mul(_mul(pad(_up(self.T, mu), (1, 0)), _dag(U[mu])), pad(self.T, (1, 0))) / 4.0
            z = dt * (4.0 / p.betasu2) * 2.0 * _mul(U[mu], s)[..., 1:]
            n = z.norm(dim=-1, keepdim=True)
            new.append(_mul(torch.cat([torch.cos(n), torch.sin(n) / n * z], -1), U[mu]))
        if self.T is not None:
            t2 = 0.5 * self.T.square().sum(-1, keepdim=True)
            force = self.triplet_staple() + (6.0 + p.msq_triplet + 2.0 * p.b4 * t2) * self.T
            if self.phi:
                force = force + p.a2 * 0.5 * self.phi[0].square().sum(-1, keepdim=True) * self.T
            self.T = self.T - dt * force
        self.U = new

    def flow(self, t_max, dt, interval):
        if self.T is not None:
            self.p.msq_triplet = self.tree_mass()
        rows, t, it = [np.concatenate([[0.0], self.measure()])], 0.0, 1
        while t < t_max:
            dt = min(dt, t_max - t) if t + dt > t_max else dt
            self.flow_step(dt)
            t += dt
            if it % interval == 0:
                rows.append(np.concatenate([[t], self.measure()]))
            it += 1
        if (it - 1) % interval:
            rows.append(np.concatenate([[t], self.measure()]))
        return np.stack(rows)

    # -- correlators --------------------------------------------------------
    def plane_ops(self, d):
        i, j = (k for k in range(3) if k != d)
        U = self.U

        def at(f, *steps):
            for k, n in steps:
                f = _up(f, k, n)
            return f

        cl = _mul(U[i], _mul(at(U[j], (i, 1)), _mul(_dag(at(U[i], (j, 1))), _dag(U[j]))))
        cl = cl + _mul(U[j], _mul(_dag(at(U[i], (j, 1), (i, -1))), _mul(_dag(at(U[j], (i, -1))), at(U[i], (i, -1)))))
        cl = cl + _mul(_dag(at(U[i], (i, -1))), _mul(_dag(at(U[j], (i, -1), (j, -1))),
                                                    _mul(at(U[i], (i, -1), (j, -1)), at(U[j], (j, -1)))))
        cl = cl + _mul(_dag(at(U[j], (j, -1))), _mul(at(U[i], (j, -1)), _mul(at(U[j], (i, 1), (j, -1)), _dag(U[i]))))
        tr = (self.T * cl[..., 1:]).sum(-1) / 4.0
        al = 2.0 * self.alpha(i, j)
        dims = tuple(k for k in range(3) if k != 2 - d)
        nx = tr.shape[2]
        x = torch.arange(nx, device=tr.device, dtype=torch.float64)
        ops = [(0.5 * self.T.square().sum(-1)).sum(dims).to(torch.complex128)]
        for f in (tr, al):
            for mom in (1, 2):
                w = torch.exp(2j * math.pi * mom * x / nx) if d != 0 else torch.ones_like(x).to(torch.complex128)
                ops.append((f * w).sum(dims))
        return ops

    def correlators(self, d):
        n, V = self.U[0].shape[2 - d], self.U[0][..., 0].numel()
        out = np.zeros((n // 2, abi.NCORR))
        ops = self.plane_ops(d)
        for r in range(n // 2):
            for k, o in enumerate(ops):
                c = (o * torch.roll(o, -r).conj()).sum() / V
                if k == 0:
                    out[r, 1] = c.real
                else:
                    out[r, 2 * k], out[r, 2 * k + 1] = c.real, c.imag
        return out

    def block(self):
        """The smeared fields of the even sites, every direction halved."""
        U, T = self.U, self.T
        new = []
        for mu in range(3):
            v = U[mu]
            for nu in range(3):
                if nu != mu:
                    v = v + _mul(U[nu], _mul(_up(U[mu], nu), _dag(_up(U[nu], mu))))
                    v = v + _up(_mul(_dag(U[nu]), _mul(U[mu], _up(U[nu], mu))), nu, -1)
            v = _mul(v, _up(v, mu))
            new.append((v / v.norm(dim=-1, keepdim=True))[::2, ::2, ::2])
        t = T
        for d in range(3):
            t = t + _rot(U[d], _up(T, d)) + _up(_rot(_dag(U[d]), T), d, -1)
        self.U, self.T = new, (t / 7.0)[::2, ::2, ::2]

    # -- one FP64 sweep -----------------------------------------------------
    def uniform(self, n, site, pass_, sweep):
        """Draw n of every site's stream: Philox4x32-10, 53 bits."""
        M = 0xFFFFFFFF
        k0, k1 = self.seed & M, self.seed >> 32
        c0, c1 = site, (pass_ << 16) | (n // 2)
        c2, c3 = torch.full_like(site, sweep), torch.full_like(site, self.chain)
        for r in range(10):
            if r:
                k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
            # the products wrap at 64 bits; their halves are taken as unsigned words
            a, b = 0xD2511F53 * c0, 0xCD9E8D57 * c2
            c0, c1, c2, c3 = ((b >> 32) & M) ^ c1 ^ k0, b & M, ((a >> 32) & M) ^ c3 ^ k1, a & M
        hi, lo = torch.where(n % 2 == 0, c0, c2), torch.where(n % 2 == 0, c1, c3)
        return ((hi << 21) | (lo >> 11)).double() * 2.0 ** -53

    def half(self, parity, mask_from, new, old):
        return torch.where((self.par == parity)[..., None] & mask_from[..., None], new, old)

    def sweep(self, seed, chain, number):
        """update_lattice with the default recipe: link heatbath, four
        overrelaxations and one Metropolis of each scalar."""
        self.seed, self.chain = seed, chain
        site = self.idx.long()
        npass = 0

        def draws():
            k = npass
            count = torch.zeros_like(site)

            def uni(where):
                u = self.uniform(count, site, k, number)
                count.add_(where.long())
                return u
            return uni

        everywhere = torch.ones_like(site, dtype=torch.bool)
        for mu in range(3):
            for parity in (0, 1):
                self.heatbath(mu, parity, draws(), everywhere)
                npass += 1
        for s in range(self.p.scalar_sweeps + 1):
            for name in ("phi", "T"):
                if not (self.phi if name == "phi" else self.T is not None):
                    continue
                for parity in (0, 1):
                    uni = draws()
                    f = self.phi[0] if name == "phi" else self.T
                    st = self.doublet_staple(0) if name == "phi" else self.triplet_staple()
                    if s < self.p.scalar_sweeps:
                        new, ok = self.overrelax(f, st, name, uni(everywhere))
                    else:
                        new, ok = self.metropolis(f, st, name, uni, everywhere)
                    f = self.half(parity, ok, new, f)
                    if name == "phi":
                        self.phi[0] = f
                    else:
                        self.T = f
                    npass += 1

    def heatbath(self, mu, parity, uni, everywhere):
        p, old = self.p, self.U[mu]
        V = -0.5 * p.betasu2 * self.staple(mu)
        for f in self.phi:
            V = V - 0.5 * _mul(_up(f, mu), _dag(f))
        norm = V.norm(dim=-1)
        V = -V / norm[..., None]
        a = 2.0 * norm
        todo, d = everywhere.clone(), torch.zeros_like(a)
        while todo.any():
            u = [uni(todo) for _ in range(4)]
            t = -torch.log(1 - u[0]) / a * torch.cos(2 * math.pi * u[2]) ** 2 - torch.log(1 - u[1]) / a
            ok = todo & ((1 - u[3]) ** 2 <= 1 - 0.5 * t)
            d = torch.where(ok, t, d)
            todo = todo & ~ok
        a0 = 1 - d
        rad = torch.sqrt(1 - a0 ** 2)
        todo, v = everywhere.clone(), torch.zeros_like(old[..., 1:])
        while todo.any():
            w = torch.stack([2 * uni(todo) - 1 for _ in range(3)], -1)
            r2 = w.square().sum(-1)
            ok = todo & (r2 <= 1) & (r2 > 0)
            v = torch.where(ok[..., None], w / torch.sqrt(r2)[..., None], v)
            todo = todo & ~ok
        new = _mul(torch.cat([a0[..., None], v * rad[..., None]], -1), _dag(V))
        ok = everywhere
        if self.T is not None:
            def hop(u):
                return -(self.T * _rot(u, _up(self.T, mu))).sum(-1)
            ok = uni(everywhere) < torch.exp(hop(old) - hop(new))
        self.U[mu] = self.half(parity, ok, new, old)

    def potential(self, name):
        """B and C of the site action f.s + B f^2 + C f^4."""
        p = self.p
        if name == "T":
            return 0.5 * p.msq_triplet + 3.0, 0.25 * p.b4
        B = 0.5 * p.msq_phi + 3.0
        if self.T is not None:
            B = B + 0.25 * p.a2 * self.T.square().sum(-1)
        return B, 0.25 * p.lambda_phi

    def overrelax(self, f, s, name, u):
        """Reflect f through the staple's direction; the component along it
        moves to the other solution of equal action."""
        B, C = self.potential(name)
        F = s.norm(dim=-1)
        e = s / F[..., None]
        X = (f * e).sum(-1)
        Y = f - X[..., None] * e
        Y2 = Y.square().sum(-1)
        b = B + 2 * Y2 * C
        c2, c1, c0 = C * X, b + C * X * X, F + b * X + C * X ** 3
        x = -c0 / c1
        for _ in range(60):  # the cubic is monotonic: Newton's method converges
            x = x - (((C * x + c2) * x + c1) * x + c0) / ((3 * C * x + 2 * c2) * x + c1)

        def dV(t):
            return F + 2 * B * t + 4 * C * (t ** 3 + Y2 * t)
        return -f + (X + x)[..., None] * e, (dV(X) / dV(x)).abs() >= u

    def metropolis(self, f, s, name, uni, everywhere):
        B, C = self.potential(name)
        if name == "T" and self.phi:
            B = B + 0.25 * self.p.a2 * self.phi[0].square().sum(-1)
        new = f + torch.stack([uni(everywhere) - 0.5 for _ in range(f.shape[-1])], -1)
        n2, f2 = new.square().sum(-1), f.square().sum(-1)
        dS = ((new - f) * s).sum(-1) + B * (n2 - f2) + C * (n2 ** 2 - f2 ** 2)
        down = dS < 0
        return new, down | (torch.exp(-dS) > uni(~down))


def exact(case, seed):
    """The outputs of `run` in 64 bits: deterministic passes of either
    precision, and FP64 sweeps of the contents whose updates are written out
    above.  The accept/reject decisions of an FP32 sweep are taken on values
    rounded to 32 bits, so its trajectory has no 64-bit counterpart."""
    kind = case["kind"]
    if kind in ("muca", "muca_pool"):
        return None
    chains = _chains(case, seed)
    params = [p for p, _ in chains]
    fields = _split(params, _host_fields(case, params, seed))
    if kind == "flow":
        lat = _Lattice64(params[0], fields[0])
        return {"rows": lat.flow(0.01 * (case["steps"] - 0.5), 0.01, case["interval"])}
    if kind == "correl":
        lat = _Lattice64(params[0], fields[0])
        sides = list(params[0].L[:3])
        d = max(range(3), key=lambda k: (sides[k], k))
        out = {"level0": lat.correlators(d)}
        for k in range(case["levels"]):
            if any(n % 2 or n <= 2 for n in sides):
                break
            sides = [n // 2 for n in sides]
            lat.block()
            out["level%d" % (k + 1)] = lat.correlators(d)
        return out
    if case["precision"] != 64 or case["content"] not in ("fund", "adj", "fundadj", "pure"):
        return None
    stored, sums = [], []
    for k, (p, chain_seed) in enumerate(chains):
        lat = _Lattice64(p, fields[k])
        for n in range(case["sweeps"]):
            lat.sweep(chain_seed, k, n)
        sums.append(lat.measure())
        if kind in ("host", "cycle"):
            stored.append(lat.stored())
    if kind == "lattice":
        return {"sums": sums[0]}
    if kind == "host":
        return stored[0]
    out = {n: np.concatenate([f[n] for f in stored]) for n in stored[0]} if stored else {}
    out["sums"] = np.stack(sums)
    return out
