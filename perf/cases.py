"""Performance cases of the force-and-step path.

Each case is one pass of work as a program that uses this package has it done: a few
engine steps with the positions and velocities read back on the device, a force
evaluation with its energies, a trip of the whole state from the host and back, the
gradient of a trajectory. `listed()` gives the standing cases, `draw()` more of the same
ranges, `prepare()` what the program holds before the pass (a started universe), `run()`
the pass and `work()` the bytes and operations it cannot do without. `exact()` restates a
case in 64-bit torch: the potentials' closed forms in place of the engine's tables, no
cells, no single precision.
"""
import ctypes
import math

import numpy as np
import torch

import mechanica_b200 as m
from mechanica_b200 import _native
from mechanica_b200 import adjoint as A
from mechanica_b200 import workloads as W

LJ = dict(lo=0.275, hi=1.0, A=9.5075e-6, B=6.1545e-3, tol=1e-3, T=10.0)
DPD = dict(alpha=25.0, gamma=4.5, sigma=3.0)
ARGON_MASS = 39.4
CHAIN = dict(bond=0.5, k_bond=100.0, k_angle=5.0, theta0=2.0, pair=(0.1, 3.0, 0.5, 1e-4, 1.5, 1e-3), radius=0.75)


def listed():
    return [
        # interactive use and the smallest example (a DPD block of 15^3): one step a call, all latency
        dict(name="dpd_3k_step", kind="dpd", n=3375, density=12.5, h=1.0, walls=True, rng="reference", steps=1),
        # the argon example as it stands: the default grid of 4^3 cells (coarser than the cutoff), a thermostat
        dict(name="argon_example_10k", kind="lj", n=10000, coarse=True, tstat=True, steps=5),
        # a larger argon fluid with cells of the cutoff and the same thermostat, a size that divides nothing
        dict(name="argon_tstat_61k", kind="lj", n=61037, coarse=False, tstat=True, steps=5),
        # the benchmark's DPD fluid: body force, no-slip walls, the reference's random term
        dict(name="dpd_200k", kind="dpd", n=200000, density=12.5, h=1.0, walls=True, rng="reference", steps=5),
        # a large DPD fluid with the counter-based random term, periodic, cells a little above the cutoff
        dict(name="dpd_1m2_philox", kind="dpd", n=1200007, density=11.0, h=1.015625, walls=False, rng="philox", steps=2),
        # a bonded solid: harmonic bonds to the six nearest neighbours with a weak Morse term, overdamped
        dict(name="bonded_32k", kind="bonded", nx=32, steps=5),
        # bead-spring chains with angles, the bonded neighbours excluded from the pair potential
        dict(name="chains_20k", kind="chains", nchains=509, length=40, steps=5),
        # an ensemble of cell-sorting replicas of mixed sizes stepped together
        dict(name="ensemble_24", kind="ensemble", nrep=24, nmin=1000, nmax=20000, steps=4),
        # chemical species carried by the particles of a fluid, with fluxes between two types
        dict(name="species_50k", kind="species", n=50021, steps=4),
        # single-point evaluation of a fluid: forces, both energies, pair virial
        dict(name="lj_energy_100k", kind="energy", n=100003, steps=1),
        # an outer program that owns the state: positions and velocities in from the host, a step, all of it out
        dict(name="roundtrip_50k", kind="roundtrip", n=50000, density=12.5, steps=1),
        # fitting potentials to a target structure: a trajectory, its loss, the gradient of both
        dict(name="adjoint_32k", kind="adjoint", n=32768, steps=8, every=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dpd", "dpd", "lj", "bonded", "chains", "ensemble", "species", "energy", "roundtrip", "adjoint"])
    if kind == "dpd":
        n = _log(rng, 1000, 1000000)
        return dict(kind=kind, n=n, density=rng.uniform(3.0, 13.0), h=1.0 + rng.randrange(0, 9) / 64.0,
                    walls=rng.random() < 0.5, rng=rng.choice(["reference", "philox"]),
                    steps=1 if n > 400000 else rng.randint(1, 5))
    if kind == "lj":
        n = _log(rng, 1000, 150000)
        return dict(kind=kind, n=n, coarse=n < 20000 and rng.random() < 0.5, tstat=rng.random() < 0.6,
                    steps=rng.randint(1, 5))
    if kind == "bonded":
        return dict(kind=kind, nx=rng.randint(8, 44), steps=rng.randint(1, 5))
    if kind == "chains":
        return dict(kind=kind, nchains=_log(rng, 30, 1500), length=rng.randint(5, 60), steps=rng.randint(1, 5))
    if kind == "ensemble":
        nmin = _log(rng, 300, 3000)
        return dict(kind=kind, nrep=rng.randint(2, 24), nmin=nmin, nmax=nmin + _log(rng, 200, 16000),
                    steps=rng.randint(1, 4))
    if kind == "species":
        return dict(kind=kind, n=_log(rng, 2000, 100000), steps=rng.randint(1, 4))
    if kind == "energy":
        return dict(kind=kind, n=_log(rng, 2000, 200000), steps=1)
    if kind == "roundtrip":
        return dict(kind=kind, n=_log(rng, 2000, 200000), density=rng.uniform(3.0, 13.0), steps=1)
    return dict(kind=kind, n=_log(rng, 2000, 32000), steps=rng.randint(2, 8), every=rng.randint(2, 4))


# ---- inputs: scenarios from the case and the seed ------------------------------------------------


def _jittered(n, L, rng, jitter=0.1):
    """n sites of a simple-cubic lattice filling a cube of edge L, jittered, as the engine takes them."""
    k = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
    g = (np.arange(k) + 0.5) * (L / k)
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    x = x[np.sort(rng.permutation(len(x))[:n])]
    x = np.mod(x + rng.uniform(-jitter, jitter, size=x.shape) * (L / k), L)
    return np.minimum(x, L * (1 - 1e-6)).astype(np.float32).astype(np.float64)


def _velocities(n, sd, rng):
    v = rng.normal(0, sd, size=(n, 3))
    return (v - v.mean(axis=0)).astype(np.float32)


def _dpd_scenario(case, seed):
    n, h = case["n"], case.get("h", 1.0)
    cells = n / case["density"]
    if case["kind"] == "roundtrip":  # a long channel
        grid = [max(3, int(round(cells / 20))), 5, 4]
    else:
        a = max(3, int(round((cells / 2) ** (1.0 / 3.0))))
        grid = [max(3, int(round(cells / (a * a)))), a, a]
    dims = [c * h for c in grid]
    scn = W.dpd(n=n, dims=dims, seed=seed)
    scn["cells"] = grid
    scn["pots"] = [("dpd", (DPD["alpha"], DPD["gamma"], DPD["sigma"], 1.0, 0), 0, 0)]
    if not case.get("walls", True):
        scn["bc"] = ("periodic",) * 3
    return scn


def _lj_scenario(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    L = (n / 10.0) ** (1.0 / 3.0)
    cells = 4 if case.get("coarse") else max(3, int(L))
    v = _velocities(n, math.sqrt(LJ["T"] / ARGON_MASS), rng)
    return dict(n=n, L=L, cells=[cells] * 3, x=_jittered(n, L, rng), v=v,
                target=0.5 * ARGON_MASS * float((v.astype(np.float64) ** 2).sum()) * 0.9, dt=0.01, tau=10.0)


def _chains_scenario(case, seed):
    """Random walks of bond-length steps turning by about pi - theta0, wrapped into a periodic cube."""
    rng = np.random.default_rng(seed)
    nc, ln, c = case["nchains"], case["length"], CHAIN
    L = max(4.0, (nc * ln / 4.0) ** (1.0 / 3.0))

    def unit(a):
        return a / np.linalg.norm(a, axis=1, keepdims=True)

    p, d = rng.uniform(0, L, size=(nc, 3)), unit(rng.normal(size=(nc, 3)))
    beads = [p]
    for _ in range(ln - 1):
        ax = unit(np.cross(d, rng.normal(size=(nc, 3))))
        turn = (np.pi - c["theta0"]) + rng.normal(0, 0.15, size=(nc, 1))
        d = unit(d * np.cos(turn) + np.cross(ax, d) * np.sin(turn))
        p = p + c["bond"] * (1 + rng.normal(0, 0.05, size=(nc, 1))) * d
        beads.append(p)
    x = np.mod(np.stack(beads, 1).reshape(-1, 3), L)
    x = np.minimum(x, L * (1 - 1e-6)).astype(np.float32).astype(np.float64)
    n = len(x)
    idx = np.arange(n, dtype=np.int32).reshape(nc, ln)
    bi, bj = idx[:, :-1].ravel().copy(), idx[:, 1:].ravel().copy()
    return dict(dim=[L] * 3, cells=[int(L)] * 3, cutoff=1.0, dt=0.002, bc=("periodic",) * 3,
                types=[(1.0, c["radius"], m.Newtonian)], pots=[("morse", c["pair"], 0, 0)], forces=[], x=x,
                v=_velocities(n, math.sqrt(0.1), rng).astype(np.float64), t=np.zeros(n, dtype=np.int32), bi=bi, bj=bj,
                bond_pot=("harmonic", (c["k_bond"], c["bond"], 0.1, 1.0, 0.009)),
                dissociation=float(np.finfo(np.float64).max), ex_i=bi.copy(), ex_j=bj.copy(),
                ai=idx[:, :-2].ravel().copy(), aj=idx[:, 1:-1].ravel().copy(), ak=idx[:, 2:].ravel().copy(),
                angle_pot=("harmonic_angle", (c["k_angle"], c["theta0"], 0.0, np.pi, 0.005 * np.pi)))


def _species_scenario(case, seed):
    scn = W.species(n=case["n"], L=max(4.0, (case["n"] / 4.0) ** (1.0 / 3.0)), seed=seed)
    scn["types"] = [(1.0, 0.7, m.Newtonian)] * 2  # the wells at r = 0.8: the fluid does not collapse
    return scn


def _ensemble_specs(case, seed):
    """Replicas of sizes spread evenly over the case's range; positions and potentials from the seed."""
    sizes = np.linspace(case["nmin"], case["nmax"], case["nrep"]).astype(int)
    return [W.cell_sorting_specs(nrep=1, seed=1000 * (seed % 1000003) + r, nmin=int(n), nmax=int(n))[0]
            for r, n in enumerate(sizes)]


class _State:
    """A started universe and the buffers its program reads results into."""

    def __init__(self, case, u):
        self.kind, self.steps, self.u = case["kind"], case["steps"], u
        u.handle  # builds and starts the engine
        n = len(u._t)
        self.x4 = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        self.v4 = torch.zeros((n, 4), dtype=torch.float32, device="cuda")

    def __del__(self):
        try:
            torch.cuda.synchronize()
            self.u.close()
        except Exception:
            pass


def _build_lj(scn, tstat):
    m.init(dim=[scn["L"]] * 3, cells=scn["cells"], cutoff=1.0, dt=scn["dt"],
           bc={"x": "periodic", "y": "periodic", "z": "periodic"})
    argon = type("Argon", (m.Particle,), {"mass": ARGON_MASS, "radius": 0.1, "target_temperature": scn["target"]})
    m.bind(m.Potential.lennard_jones_12_6(LJ["lo"], LJ["hi"], LJ["A"], LJ["B"], LJ["tol"]), argon, argon)
    if tstat:
        m.bind(m.forces.berenderson_tstat(scn["tau"]), argon)
    argon.factory(positions=scn["x"], velocities=scn["v"])
    return m.universe


def prepare(case, seed):
    m.universe = type(m.universe)()  # several states are alive at once, each with a universe of its own
    kind = case["kind"]
    if kind == "dpd":
        return _State(case, W.build_gpu(_dpd_scenario(case, seed), rng_mode=case["rng"]))
    if kind in ("lj", "energy"):
        return _State(case, _build_lj(_lj_scenario(case, seed), case.get("tstat", False)))
    if kind == "bonded":
        return _State(case, W.build_bonded_adjoint(W.bonded_block(nx=case["nx"], seed=seed))[0])
    if kind == "chains":
        return _State(case, W.build_gpu(_chains_scenario(case, seed)))
    if kind == "ensemble":
        return _State(case, W.build_gpu_batch(_ensemble_specs(case, seed)))
    if kind == "species":
        return _State(case, W.build_gpu(_species_scenario(case, seed)))
    if kind == "roundtrip":
        scn = _dpd_scenario(case, seed)
        s = _State(case, W.build_gpu(scn))
        s.x, s.v = scn["x"], scn["v"].astype(np.float32)
        return s
    spec = W.adjoint_spec(n=case["n"], seed=seed)
    u, params = W.build_adjoint(spec)
    s = _State(case, u)
    s.sim = A.Simulation(u, params, case["steps"], checkpoint_every=case["every"])
    s.theta = torch.tensor(params.theta(), dtype=torch.float32, requires_grad=True)
    s.x0 = torch.tensor(spec["x"], dtype=torch.float32, requires_grad=True)
    s.v0 = torch.tensor(spec["v"], dtype=torch.float32, requires_grad=True)
    s.target = torch.tensor(W.rdf_target(), device="cuda")
    s.box = spec["dim"]
    s.counts = (int((spec["t"] == 0).sum()), int((spec["t"] == 1).sum()))
    return s


def run(s):
    u = s.u
    if s.kind == "energy":
        u.force()
        ep, ek = u.energies()
        return {"forces": u.forces, "virial": u.virial(), "epot": ep, "ekin": ek}
    if s.kind == "roundtrip":
        u.load(s.x, s.v)
        u.steps(s.steps)
        x, v, f, cell, xrel = u.state()
        return {"x": x, "v": v, "f": f, "cell": cell, "xrel": xrel}
    if s.kind == "adjoint":
        x4 = A.trajectory(s.theta, s.x0, s.v0, s.sim)
        loss, g = A.rdf_loss(x4, s.target, s.box, 0, 1, counts=s.counts)
        grads = torch.autograd.grad(loss, (s.theta, s.x0, s.v0))
        # the radial distribution in the precision of the positions it is taken from
        return {"x": x4.detach(), "loss": loss.detach().float(), "g": g.detach().float(), "theta": grads[0], "x0": grads[1],
                "v0": grads[2]}
    u.steps(s.steps)
    p = [ctypes.c_void_p(t.data_ptr()) for t in (s.x4, s.v4)]
    _native.check(_native.lib().mxg_engine_positions(u.handle, p[0], p[1]), "positions")
    out = {"x": s.x4, "v": s.v4}
    if s.kind == "species":
        out["species"] = u.species_values()
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------


def _sizes(case):
    """(particles, interacting pairs a force pass, operations a pair)."""
    k = case["kind"]
    sphere = 4.0 / 3.0 * math.pi
    if k in ("dpd", "roundtrip"):
        return case["n"], 0.5 * sphere * case["density"] / case.get("h", 1.0) ** 3 * case["n"], 40
    if k in ("lj", "energy"):
        return case["n"], 0.5 * sphere * 10.0 * case["n"], 44
    if k == "bonded":
        n = case["nx"] ** 3
        return n, 13 * n, 44
    if k == "chains":
        n = case["nchains"] * case["length"]
        return n, 0.5 * sphere * 4.0 * n + 3 * n, 44
    if k == "ensemble":
        n = case["nrep"] * (case["nmin"] + case["nmax"]) // 2
        return n, 0.5 * sphere * 2.5 ** 3 * 0.8 * n, 44
    if k == "species":
        return case["n"], 0.5 * sphere * 4.0 * case["n"], 64
    return case["n"], 0.5 * sphere * 2.5 ** 3 * 0.8 * case["n"], 84


def work(case):
    n, pairs, ops = _sizes(case)
    k, steps = case["kind"], case["steps"]
    state = 32.0 * n  # positions and velocities, float4 each
    if k == "energy":
        return {"bytes": state + 12.0 * n, "flops": pairs * (ops + 20)}
    if k == "roundtrip":
        return {"bytes": 36.0 * n + 2 * state + 64.0 * n, "flops": pairs * ops}
    if k == "adjoint":  # forward, and per step back its force pass again and the two-sided derivative
        return {"bytes": steps * 6 * state, "flops": steps * pairs * ops * 4}
    return {"bytes": steps * 2 * state + state, "flops": steps * (pairs * ops + 20.0 * n)}


# ---- the cases in 64 bits -------------------------------------------------------------------------


def _pairs(x, box, periodic, rc):
    """(i, j, x_i - x_j) of the pairs i != j within rc, once each; x inside the box, (N, 3) float64."""
    dev = x.device
    box_t = torch.tensor(box, dtype=torch.float64, device=dev)
    nc = [max(1, int(b / rc)) for b in box]
    nc = [k if k >= 3 else 1 for k in nc]
    nct = torch.tensor(nc, device=dev)
    c3 = torch.minimum((x.detach() / box_t * nct).long().clamp_(min=0), nct - 1)
    cell = (c3[:, 0] * nc[1] + c3[:, 1]) * nc[2] + c3[:, 2]
    order = torch.argsort(cell, stable=True)
    ncell = nc[0] * nc[1] * nc[2]
    count = torch.bincount(cell, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    K = int(count.max())
    tab = torch.full((ncell, K), -1, dtype=torch.long, device=dev)
    rank = torch.arange(len(x), device=dev) - start[cell[order]]
    tab[cell[order], rank] = order
    xp = torch.full((ncell, K, 3), float("nan"), dtype=torch.float64, device=dev)
    xp[cell[order], rank] = x.detach()[order]
    loc = torch.stack([torch.arange(ncell, device=dev) // (nc[1] * nc[2]),
                       torch.arange(ncell, device=dev) // nc[2] % nc[1], torch.arange(ncell, device=dev) % nc[2]], 1)
    ranges = [(-1, 0, 1) if k > 1 else (0,) for k in nc]
    offsets = [(a, b, c) for a in ranges[0] for b in ranges[1] for c in ranges[2] if (a, b, c) >= (0, 0, 0)]
    per = torch.tensor([1.0 if p else 0.0 for p in periodic], dtype=torch.float64, device=dev)
    chunk = max(1, int(3e7 // (K * K)))
    found = []
    for off in offsets:
        other = loc + torch.tensor(off, device=dev)
        ok = torch.ones(ncell, dtype=torch.bool, device=dev)
        for q in range(3):
            if not periodic[q]:
                ok &= (other[:, q] >= 0) & (other[:, q] < nc[q])
        other = other % nct
        oc = (other[:, 0] * nc[1] + other[:, 1]) * nc[2] + other[:, 2]
        cells = torch.nonzero(ok).ravel()
        for k0 in range(0, len(cells), chunk):
            c = cells[k0:k0 + chunk]
            r2 = 0.0
            for q in range(3):
                d = xp[c][:, :, None, q] - xp[oc[c]][:, None, :, q]
                d = d - per[q] * box[q] * torch.round(d / box[q])
                r2 = r2 + d * d
            hit = r2 <= rc * rc
            if off == (0, 0, 0):
                hit &= torch.ones((K, K), dtype=torch.bool, device=dev).triu(1)
            b, p, q = torch.nonzero(hit, as_tuple=True)
            found.append(torch.stack([tab[c[b], p], tab[oc[c[b]], q]]))
    ij = torch.cat(found, 1)
    i, j = ij[0], ij[1]
    d = x[i] - x[j]
    return i, j, d - per * box_t * torch.round(d.detach() / box_t)


def _scatter(n, i, j, f):
    """Sum of f on i and of -f on j."""
    out = torch.zeros((n, 3), dtype=torch.float64, device=f.device)
    return out.index_add(0, i, f).index_add(0, j, -f)


def _morse(p, r, ri, rj):
    """(energy, dV/dr, range mask) of the shifted Morse potential p = (d, a, r0, min, max, tol)."""
    s = r - (ri + rj) + p[2] + 1.0
    e = torch.exp(-p[1] * (s - 1.0))
    ok = s <= p[4]
    return torch.where(ok, p[0] * (e * e - 2 * e), 0 * e), torch.where(ok, 2 * p[0] * p[1] * (e - e * e), 0 * e), ok


def _lj(r):
    i6 = r ** -6
    return LJ["A"] * i6 * i6 - LJ["B"] * i6, (-12 * LJ["A"] * i6 * i6 + 6 * LJ["B"] * i6) / r


def _philox_xi(step, a, b):
    """The pair random number: Philox4x32-10 keyed on (step, ids), uniform of unit variance."""
    m32 = 0xFFFFFFFF
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    c = [lo.clone(), hi.clone(), torch.full_like(lo, step & m32), torch.full_like(lo, step >> 32)]
    k = [0x44504431, 0x58495F31]

    def mul(w, v):  # 32 x 32 -> (high, low) words in signed 64-bit arithmetic
        p0, p1 = w * (v & 0xFFFF), w * (v >> 16)
        t = p1 + (p0 >> 16)
        return t >> 16, ((t & 0xFFFF) << 16) | (p0 & 0xFFFF)

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k[0], l1, h0 ^ c[3] ^ k[1], l0]
        k = [(k[0] + 0x9E3779B9) & m32, (k[1] + 0xBB67AE85) & m32]
    u = ((c[0] >> 8).double() + 0.5) / 16777216.0
    return math.sqrt(3.0) * (2 * u - 1)


def _dpd_force(d, r, w, alpha, gamma, sigma, rc, dt, xi):
    """Force on the pair's first particle."""
    om = 1 - r / rc
    e = d / r[:, None]
    f = alpha * om - gamma * om * om * (e * w).sum(1) + sigma * om / math.sqrt(dt) * xi
    return f[:, None] * e


def _clamp(v, top):
    return torch.minimum(torch.maximum(v, -top), top)


def _cuda(a):
    return torch.tensor(np.asarray(a), dtype=torch.float64, device="cuda")


def _advance(x, v, f, mass, dt, h, box, bc, overdamped):
    """Forward Euler with the speed (or step) limit, no-slip walls and the periodic wrap."""
    h = _cuda(h)
    if overdamped:
        x = x + _clamp(dt * f / mass, h * 0.05)
    else:
        v = _clamp(v + dt * f / mass, h * 0.05 / dt)
        x = x + dt * v
    for q in range(3):
        if bc[q] == "periodic":
            x = torch.cat([x[:, :q], x[:, q:q + 1] - box[q] * torch.floor(x[:, q:q + 1].detach() / box[q]), x[:, q + 1:]], 1)
        else:
            low, high = x[:, q] <= 0, x[:, q] >= box[q]
            out = (low | high)[:, None]
            xq = torch.where(low, -x[:, q], torch.where(high, 2 * box[q] - x[:, q], x[:, q]))
            x = torch.cat([x[:, :q], xq[:, None], x[:, q + 1:]], 1)
            v = torch.where(out, -v, v)
    return x, v


def _with_bits(a, bits):
    """(N, 4): a and the integer bits as the engine carries them in w."""
    w = torch.as_tensor(np.asarray(bits, dtype=np.int32)).view(torch.float32).double().cuda()
    return torch.cat([a, w[:, None]], 1)


def _scenario_run(scn, steps, force, observe=None):
    """steps of a scenario dict under force(x, v, step, box) -> (N, 3)."""
    box, dt = [float(b) for b in scn["dim"]], float(np.float32(scn["dt"]))
    h = [b / c for b, c in zip(box, scn["cells"])]
    mass, _, dyn = scn["types"][0]
    x, v = _cuda(scn["x"]), _cuda(np.asarray(scn["v"], dtype=np.float32))
    for s in range(steps):
        f = force(x, v, s, box)
        x0 = x
        x, v = _advance(x, v, f, mass, dt, h, box, scn["bc"], dyn == m.Overdamped)
        if observe:
            observe(x0, x, dt, h)
    return x, v


def _dpd_exact_force(scn, rng):
    periodic = [b == "periodic" for b in scn["bc"]]
    body = _cuda(scn["forces"][0][1:]) if scn["forces"] else 0.0
    alpha, gamma, sigma, rc = scn["pots"][0][1][:4]

    def force(x, v, step, box):
        i, j, d = _pairs(x, box, periodic, rc)
        xi = _philox_xi(step, i, j) if rng == "philox" else 1.0
        f = _dpd_force(d, d.norm(dim=1), v[i] - v[j], alpha, gamma, sigma, rc, scn["dt"], xi)
        return _scatter(len(x), i, j, f) + body

    return force


def _morse_pairs_force(scn):
    """Morse per type pair (and nothing else), as W.cell_sorting_specs, W.species and the chains have it."""
    t = torch.as_tensor(scn["t"]).long().cuda()
    radius = scn["types"][0][1]
    table = {(a, b): p for (_, p, a, b) in scn["pots"]}

    def force(x, v, step, box):
        i, j, d = _pairs(x, box, [True] * 3, scn["cutoff"])
        r = d.norm(dim=1)
        dv = torch.zeros_like(r)
        for (a, b), p in table.items():
            hit = ((t[i] == a) & (t[j] == b)) | ((t[i] == b) & (t[j] == a))
            dv = torch.where(hit, _morse(p, r, radius, radius)[1], dv)
        return _scatter(len(x), i, j, -(dv / r)[:, None] * d)

    return force


def _bond_force(x, bi, bj, box, k, r0, lo, hi):
    L = _cuda(box)
    d = x[bi] - x[bj]
    d = d - L * torch.round(d / L)
    rc = d.norm(dim=1).clamp(lo, hi)
    return _scatter(len(x), bi, bj, -(2 * k * (rc - r0) / rc)[:, None] * d)


def _exact_lj(case, seed):
    scn = _lj_scenario(case, seed)
    box, dt = [scn["L"]] * 3, float(np.float32(scn["dt"]))

    def force(x, v):
        i, j, d = _pairs(x, box, [True] * 3, 1.0)
        r = d.norm(dim=1)
        e, dv = _lj(r)
        fp = -(dv / r)[:, None] * d
        return e.sum(), d.T @ fp, _scatter(len(x), i, j, fp)

    x, v = _cuda(scn["x"]), _cuda(scn["v"])
    if case["kind"] == "energy":
        e, w, f = force(x, v)
        return {"forces": f, "virial": w, "epot": e, "ekin": 0.5 * ARGON_MASS * (v * v).sum()}
    h = [scn["L"] / c for c in scn["cells"]]
    for _ in range(case["steps"]):
        f = force(x, v)[2]
        if case["tstat"]:
            f = f + (scn["target"] / (0.5 * ARGON_MASS * (v * v).sum()) - 1) / scn["tau"] * v
        x, v = _advance(x, v, f, ARGON_MASS, dt, h, box, ("periodic",) * 3, False)
    n = scn["n"]
    return {"x": _with_bits(x, np.zeros(n)), "v": _with_bits(v, np.arange(n))}


def _exact_bonded(case, seed):
    spec = W.bonded_block(nx=case["nx"], seed=seed)
    rad, (k, r0, lo, hi, _) = spec["radius"], spec["harmonic"]
    bi, bj = (torch.as_tensor(spec[q]).long().cuda() for q in ("bi", "bj"))
    scn = dict(spec, v=np.zeros_like(spec["x"]), types=[(1.0, rad, m.Overdamped)])

    def force(x, v, step, box):
        i, j, d = _pairs(x, box, [True] * 3, spec["cutoff"])
        r = d.norm(dim=1)
        dv = _morse(spec["morse"], r, rad, rad)[1]
        return _scatter(len(x), i, j, -(dv / r)[:, None] * d) + _bond_force(x, bi, bj, box, k, r0, lo, hi)

    x, v = _scenario_run(scn, case["steps"], force)
    return {"x": _with_bits(x, spec["t"]), "v": _with_bits(v, np.arange(len(spec["x"])))}


def _exact_chains(case, seed):
    scn = _chains_scenario(case, seed)
    c, p, rad = CHAIN, CHAIN["pair"], CHAIN["radius"]
    bi, bj, ai, aj, ak = (torch.as_tensor(scn[q]).long().cuda() for q in ("bi", "bj", "ai", "aj", "ak"))
    pair = _morse_pairs_force(scn)

    def unshifted(r):  # what an exclusion takes back: the pair's table without the radii shift
        e = torch.exp(-p[1] * (r - 1.0))
        return 2 * p[0] * p[1] * (e - e * e)

    def force(x, v, step, box):
        L = _cuda(box)
        f = pair(x, v, step, box) + _bond_force(x, bi, bj, box, c["k_bond"], c["bond"], 0.1, 1.0)
        d = x[bi] - x[bj]
        d = d - L * torch.round(d / L)
        r = d.norm(dim=1)
        f = f + _scatter(len(x), bi, bj, torch.where(r <= 1.0, unshifted(r) / r, 0 * r)[:, None] * d)
        if len(ai):
            y = x.detach().requires_grad_(True)
            u, w = y[ai] - y[aj], y[ak] - y[aj]
            u, w = u - L * torch.round(u.detach() / L), w - L * torch.round(w.detach() / L)
            th = torch.acos(((u * w).sum(1) / (u.norm(dim=1) * w.norm(dim=1))).clamp(-1 + 1e-12, 1 - 1e-12))
            f = f - torch.autograd.grad((c["k_angle"] * (th - c["theta0"]) ** 2).sum(), y)[0]
        return f

    x, v = _scenario_run(scn, case["steps"], force)
    return {"x": _with_bits(x, scn["t"]), "v": _with_bits(v, np.arange(len(scn["x"])))}


def _exact_ensemble(case, seed):
    xs, vs, ts = [], [], []
    for scn in _ensemble_specs(case, seed):
        x, v = _scenario_run(scn, case["steps"], _morse_pairs_force(scn))
        xs.append(x)
        vs.append(v)
        ts.append(scn["t"])
    t = np.concatenate(ts)
    return {"x": _with_bits(torch.cat(xs), t), "v": _with_bits(torch.cat(vs), np.arange(len(t)))}


def _exact_species(case, seed):
    scn = _species_scenario(case, seed)
    t = torch.as_tensor(scn["t"]).long().cuda()
    box = [float(b) for b in scn["dim"]]
    s = _cuda(scn["sp_values"])
    rate = torch.zeros_like(s)

    def one(kind, k, target, sa, sb):
        if kind == 0:
            return k * (sa - sb)
        u = k * (sa - target) if kind == 1 else k * (target - sb) * sa
        return u.clamp(min=0)

    def observe(x0, x1, dt, h):
        nonlocal s, rate
        i, j, d = _pairs(x0, box, [True] * 3, scn["cutoff"])
        w = (1 - d.norm(dim=1) / scn["cutoff"]) ** 2
        for (kind, ta, tb, ia, ib, k, decay, target) in scn["fluxes"]:
            for a, b in ((i, j),) if ta == tb else ((i, j), (j, i)):
                hit = (t[a] == ta) & (t[b] == tb)
                p, q = a[hit], b[hit]
                qq = w[hit] * one(kind, k, target, s[p, ia], s[q, ib])
                rate[:, ia] = rate[:, ia].index_add(0, p, -qq - 0.5 * decay * s[p, ia])
                rate[:, ib] = rate[:, ib].index_add(0, q, qq - 0.5 * decay * s[q, ib])
        ht, grid = _cuda(h), torch.tensor(scn["cells"], device="cuda")
        kept = ((x0 / ht).long() % grid == (x1 / ht).long() % grid).all(1, keepdim=True)
        konst = torch.as_tensor((scn["sp_flags"][scn["t"]] & 4) != 0).cuda()
        s = torch.where(kept & ~konst, s + scn["dt"] * rate, s)
        rate = torch.where(kept, torch.zeros_like(rate), rate)

    x, v = _scenario_run(scn, case["steps"], _morse_pairs_force(scn), observe)
    return {"x": _with_bits(x, scn["t"]), "v": _with_bits(v, np.arange(len(scn["x"]))), "species": s}


def _exact_adjoint(case, seed):
    spec = W.adjoint_spec(n=case["n"], seed=seed)
    n, box, dt, rc = case["n"], [float(b) for b in spec["dim"]], float(np.float32(spec["dt"])), spec["cutoff"]
    t = torch.as_tensor(spec["t"]).long().cuda()
    _, gamma, sigma, _, _ = spec["dpd"]
    theta0 = np.concatenate([np.asarray(q[:3]) for q in spec["morse"].values()] + [[gamma]]).astype(np.float32)
    theta = _cuda(theta0).requires_grad_(True)
    x0 = _cuda(np.asarray(spec["x"], dtype=np.float32)).requires_grad_(True)
    v0 = _cuda(spec["v"]).requires_grad_(True)
    h = [b / c for b, c in zip(box, spec["cells"])]
    radius = spec["types"][0][1]
    x, v = x0, v0
    for s in range(case["steps"]):
        i, j, d = _pairs(x, box, [True] * 3, rc)
        r = d.norm(dim=1)
        kind = (t[i] + t[j]).clamp(max=2)
        q = theta[:9].reshape(3, 3)[kind]
        s1 = r - 2 * radius + q[:, 2]  # the table's argument less one
        e = torch.exp(-q[:, 1] * s1)
        ok = s1.detach() + 1.0 <= rc
        fm = torch.where(ok, -2 * q[:, 0] * q[:, 1] * (e - e * e) / r, 0 * r)[:, None] * d
        f = fm + _dpd_force(d, r, v[i] - v[j], 0.0, theta[9], sigma, rc, spec["dt"], _philox_xi(s, i, j))
        x, v = _advance(x, v, _scatter(n, i, j, f), 1.0, dt, h, box, spec["bc"], False)
    nb, rmax = 64, 2.5
    dr = rmax / nb
    c = (torch.arange(nb, dtype=torch.float64, device="cuda") + 0.5) * dr
    i, j, d = _pairs(x, box, [True] * 3, rmax + 4 * dr)
    hit = t[i] != t[j]
    r = d[hit].norm(dim=1)
    near = (r.detach() / dr - 0.5).round().long()
    hist = torch.zeros(nb, dtype=torch.float64, device="cuda")
    gauss = 1 / (math.sqrt(2 * math.pi) * dr)
    for o in range(-5, 6):  # a Gaussian of one bin's width, minus its value at the cut of four
        b = near + o
        u = (r - (b.double() + 0.5) * dr) / dr
        use = (b >= 0) & (b < nb) & (u.detach().abs() <= 4)
        hist = hist.index_add(0, b[use], gauss * (torch.exp(-0.5 * u[use] ** 2) - math.exp(-8.0)))
    g = hist * (float(np.prod(box)) / (float((t == 0).sum()) * float((t == 1).sum())) / (4 * math.pi * c ** 2))
    loss = ((g - _cuda(W.rdf_target())) ** 2).sum()
    grads = torch.autograd.grad(loss, (theta, x0, v0))
    return {"x": _with_bits(x.detach(), spec["t"]), "loss": loss.detach(), "g": g.detach(), "theta": grads[0],
            "x0": grads[1], "v0": grads[2]}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("lj", "energy"):
        return _exact_lj(case, seed)
    if kind in ("bonded", "chains", "ensemble", "species", "adjoint"):
        return {"bonded": _exact_bonded, "chains": _exact_chains, "ensemble": _exact_ensemble,
                "species": _exact_species, "adjoint": _exact_adjoint}[kind](case, seed)
    scn = _dpd_scenario(case, seed)
    n = case["n"]
    force = _dpd_exact_force(scn, case.get("rng", "reference"))
    if kind == "roundtrip":
        x0, v0 = _cuda(scn["x"]), _cuda(scn["v"])
        box, dt, h = [float(b) for b in scn["dim"]], float(np.float32(scn["dt"])), _cuda([1.0] * 3)
        f = force(x0, v0, 0, box)
        x, v = _advance(x0, v0, f, 1.0, dt, [1.0] * 3, box, scn["bc"], False)
        grid = torch.tensor(scn["cells"], device="cuda")
        c = torch.minimum((x / h).long(), grid - 1)
        # the cell index is a whole number, compared as such
        return {"x": x, "v": v, "f": f, "cell": None, "xrel": x - c * h}
    x, v = _scenario_run(scn, case["steps"], force)
    return {"x": _with_bits(x, np.zeros(n)), "v": _with_bits(v, np.arange(n))}
