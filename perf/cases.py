"""Performance cases of the framework: what programs built on it have it do.

A case is a dict of plain values naming a kind of call, a seeded box and the
call's options.  The kinds, all through the public entry points
(``quantom_b200.engine.Engine``, ``quantom_b200.grad.trajectory_loss``):

* ``drive``      one step at a time, errors surfaced and positions read after
                 each (the reference's own driver loop: deviceMaster,
                 hostMaster, then the display's positions);
* ``md``         a stretch of molecular dynamics between two trajectory
                 frames: n steps, then the unwrapped positions;
* ``log``        the same with every step's energies recorded and read back
                 (drift and temperature monitoring);
* ``evaluate``   forces and energies of given coordinates (labelling, an
                 external sampler): state in, one evaluation, results out;
* ``grad``       one optimisation step of force-field parameters: trajectory
                 loss and its gradient through ``torch.autograd``;
* ``loss``       the forward half alone (a line search, a validation loss);
* ``reference``  the same stretch of dynamics in the reference's own
                 semantics (parity studies), its lists every 200 steps and
                 its thermostat every 40;
* ``render``     the picture of the current state.

Boxes are the repository's synthetic ones (LJ waters at liquid density, bead
chains of up to 64 particles per compound): packed once per size, then every
seed shifts the whole box by a random vector and draws its own
Maxwell-Boltzmann velocities.  ``exact`` restates the physics in FP64 with
plain torch.
"""
import functools
import math

import numpy as np
import torch

from quantom_b200 import engine as E
from quantom_b200 import grad as G
from quantom_b200 import layout as L
from quantom_b200 import systems as S

R_GAS = 8.314462618


def _case(name, kind, box, waters, chains=0, length=0, steps=1, precision="fp32", thermostat="none", cutoff=1.2,
          skin=0.1, checkpoint=0):
    c = dict(kind=kind, box=box, waters=waters, chains=chains, length=length, steps=steps, precision=precision,
             thermostat=thermostat, cutoff=cutoff, skin=skin, checkpoint=checkpoint)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest box, one step per call: launch and synchronisation latency of an interactive driver
        _case("drive_waters_880", "drive", 3.0, 880),
        # the neat water box at constant energy, frames every 200 steps
        _case("nve_waters_4096", "md", 5.0, 4096, steps=200),
        # a solvated, bridged pair of chains with an odd particle count, thermostatted, energies of every step
        _case("log_bridged_3893", "log", 5.0, 3701, 2, 96, steps=200, thermostat="berendsen"),
        # the benchmark box, plain FP32 with a thermostat: the everyday production run
        _case("nvt_chains_32k", "md", 10.0, 31000, 16, 64, steps=200, thermostat="berendsen"),
        # the same box in mixed precision at constant energy: long drift-free runs
        _case("nve_mixed_chains_32k", "md", 10.0, 31000, 16, 64, steps=200, precision="mixed"),
        # the largest box: two compounds and a bridge per chain, 32-bit list ids
        _case("nvt_mixed_chains_258k", "md", 20.0, 250000, 64, 128, steps=60, precision="mixed",
              thermostat="berendsen"),
        # one labelled configuration of the benchmark box
        _case("evaluate_chains_32k", "evaluate", 10.0, 31000, 16, 64),
        # the learning path: 200 unrolled steps, checkpoints every 20 (forward and backward)
        _case("grad_waters_8192", "grad", 6.3, 8192, steps=200, skin=0.2, checkpoint=20),
        # gradients of bonded and non-bonded parameters of a small solvated chain box
        _case("grad_chains_1948", "grad", 4.0, 1900, 2, 24, steps=50, skin=0.2, checkpoint=10),
        # a validation loss: the forward half
        _case("loss_waters_8192", "loss", 6.3, 8192, steps=200, skin=0.2, checkpoint=20),
        # the reference's own semantics on the benchmark box
        _case("reference_chains_32k", "reference", 10.0, 31000, 16, 64, steps=200, thermostat="reference"),
        # a frame of the display of the benchmark box
        _case("render_chains_32k", "render", 10.0, 31000, 16, 64),
    ]


def draw(rng):
    """One more case: sizes over the whole range (their logarithm), odd counts, every kind."""
    kind = rng.choices(["drive", "md", "log", "evaluate", "grad", "loss", "reference", "render"],
                       [1, 5, 1, 1, 2, 1, 1, 1])[0]
    top = {"drive": 60000, "md": 240000, "log": 60000, "evaluate": 60000, "grad": 9000, "loss": 9000,
           "reference": 32000, "render": 60000}[kind]
    n = int(math.exp(rng.uniform(math.log(900), math.log(top))))
    box = round((n / 32.5) ** (1.0 / 3.0) + 0.02, 3)
    chains, length = 0, 0
    if rng.random() < 0.6 and n > 1500:
        # a compound has to fit the box (its extent below 0.45 of the side)
        length = rng.randint(5, 24) if box < 4.9 else rng.randint(5, 64 if box < 9.5 or kind == "reference" else 128)
        chains = rng.randint(1, max(1, min(24, n // (12 * length))))
    cutoff = rng.choice([1.0, 1.2, 1.2, 1.4]) if kind != "reference" else 1.2
    skin = 0.2 if kind in ("grad", "loss") else 0.1
    if 2.0 * (cutoff + skin) > 0.98 * box:
        cutoff = 1.2
    steps = {"drive": 1, "evaluate": 1, "render": 1}.get(kind) or rng.randint(40, 160)
    if kind == "md":
        steps = max(20, min(steps, int(60 * 250000 / n)))
    precision = rng.choice(["fp32", "mixed"]) if kind in ("drive", "md", "log", "evaluate") else "fp32"
    thermostat = "reference" if kind == "reference" else "none"
    if kind in ("drive", "md", "log") and rng.random() < 0.5:
        thermostat = "berendsen"
    return _case(None, kind, box, n - chains * length, chains, length, steps, precision, thermostat, cutoff, skin,
                 rng.randint(7, 25) if kind in ("grad", "loss") else 0)


# ---------------------------------------------------------------- inputs ---
@functools.lru_cache(maxsize=8)
def _packed(box, waters, chains, length):
    spec = S.SystemSpec("box", box, waters, chains=S.ChainSpec(chains, length) if chains else None,
                        mc_sweeps=30 if waters < 50000 else 6)
    return S.make_system(spec, seed=2024)


def _system(case, seed):
    """The packed box shifted by a random vector, with its own velocities."""
    base = _packed(case["box"], case["waters"], case["chains"], case["length"])
    rng = np.random.default_rng([seed, 77])
    box, dt = base.spec.box_len, base.spec.dt
    s = base.copy()
    shift = rng.uniform(0.0, box, 3)
    mass = s.forcefield["particle_parameters"][0]["mass"].astype(np.float64)

    def velocities(types):
        v = rng.normal(size=types.shape + (3,))
        return v * np.sqrt(R_GAS * 300.0 / mass[types])[..., None]

    x = np.mod(base.solvents["pos"].astype(np.float64) + shift, box)
    v = velocities(np.zeros(len(x), np.int64))
    v -= v.mean(axis=0)
    s.solvents["pos"] = x
    s.solvents["pos_tsub1"] = x - v * dt
    if s.n_compounds:
        live = np.arange(L.MAX_COMPOUND_PARTICLES)[None, :] < base.compounds["n_particles"][:, None]
        x = base.states["positions"].astype(np.float64) + shift
        x -= np.floor(x[:, :1] / box) * box          # particle 0 of each compound inside the box
        v = velocities(base.compounds["atom_types"].astype(np.int64))
        s.states["positions"] = np.where(live[..., None], x, 0.0)
        s.compounds["prev_positions"] = np.where(live[..., None], x - v * dt, 0.0)
    return s


def _engine(case, system):
    spec = system.spec
    if case["kind"] == "reference":
        return E.Engine(system, E.default_params(box_len=spec.box_len, cutoff=case["cutoff"], dt=spec.dt,
                                                 thermostat=E.THERMOSTAT_REFERENCE, t_target=300.0))
    return E.Engine(system, E.default_params(
        box_len=spec.box_len, cutoff=case["cutoff"], dt=spec.dt, semantics=E.SEMANTICS_PHYSICS,
        precision=E.PRECISION_MIXED if case["precision"] == "mixed" else E.PRECISION_FP32, skin=case["skin"],
        switch_on=case["cutoff"] - 0.2, nlist_period=0, t_target=300.0, tau_t=1e-4,
        thermostat=E.THERMOSTAT_BERENDSEN if case["thermostat"] == "berendsen" else E.THERMOSTAT_NONE))


def _loss_spec(case):
    """U/N plus 100 x the RDF-bin loss over 50 bins ending at the cutoff, against a smooth liquid-like target."""
    bins = 50
    r_max = case["cutoff"] * bins / (bins + 1)
    r = (np.arange(bins) + 0.5) * (r_max / bins)
    n = case["waters"] + case["chains"] * case["length"]
    g = 1.0 / (1.0 + np.exp(-(r - 0.29) / 0.012)) * (1.0 + 1.6 * np.exp(-(((r - 0.34) / 0.035) ** 2)))
    target = 2.0 * math.pi * r * r * (r_max / bins) * n / case["box"] ** 3 * g
    return dict(n_steps=case["steps"], checkpoint_every=case["checkpoint"], n_bins=bins, r_max=r_max, w_energy=1.0,
                w_rdf=100.0, target=target)


def _start(system):
    return (system.states["positions"].copy() if system.n_compounds else np.zeros((0, 64, 3), np.float32),
            system.solvents["pos"].copy())


def prepare(case, seed):
    system = _system(case, seed)
    eng = _engine(case, system)
    st = dict(case=case, engine=eng, box=np.float32(system.spec.box_len), start=_start(system), frames=0)
    if case["kind"] == "log":
        eng.log_start(1, ring_frames=64, flags=0)
    elif case["kind"] == "evaluate":
        st["state"] = (system.states, np.ascontiguousarray(system.compounds["prev_positions"]), system.solvents)
    elif case["kind"] in ("grad", "loss"):
        st["spec"] = _loss_spec(case)
        theta = torch.tensor(eng.get_params(), dtype=torch.float32)
        st["theta"] = theta.requires_grad_(case["kind"] == "grad")
    return st


# ------------------------------------------------------------- the passes ---
def _unwrapped(st):
    """Positions in the image nearest the run's first frame (diffusion and contact analyses need no box jumps)."""
    out = []
    for x, x0 in zip(st["engine"].positions(), st["start"]):
        k = np.subtract(x, x0)
        k *= np.float32(1.0) / st["box"]
        np.rint(k, out=k)
        k *= st["box"]
        x -= k
        out.append(x)
    return out


def run(st):
    case, eng = st["case"], st["engine"]
    kind = case["kind"]
    if kind == "drive":
        eng.deviceMaster()
        eng.hostMaster()
        return _unwrapped(st)
    if kind in ("md", "reference"):
        eng.step(case["steps"])
        return _unwrapped(st)
    if kind == "log":
        eng.step(case["steps"])
        frames = eng.log_read(st["frames"])
        st["frames"] += case["steps"]
        # the sums' addends (pair and bonded terms, FP32 velocities) are FP32: the monitor keeps FP32
        return _unwrapped(st) + [frames["energies"].astype(np.float32)]
    if kind == "evaluate":
        eng.set_state(*st["state"])
        energies = eng.compute_energies()
        return list(eng.forces()) + [energies.astype(np.float32)]
    if kind == "grad":
        theta = st["theta"]
        theta.grad = None
        loss = G.trajectory_loss(theta, eng, **st["spec"])
        loss.backward()
        return [loss.detach(), theta.grad]
    if kind == "loss":
        return [G.trajectory_loss(st["theta"], eng, **st["spec"])]
    return [eng.render_image(1080, 1080)]


def work(case):
    """The state read once (positions and previous positions) and each output written once; per step 32 FLOP a
    unique pair within the cutoff, and for a gradient the same pairs' second derivatives (96 FLOP)."""
    n = case["waters"] + case["chains"] * case["length"]
    pairs = 0.5 * n * (n / case["box"] ** 3) * 4.0 / 3.0 * math.pi * case["cutoff"] ** 3
    kind = case["kind"]
    if kind == "render":
        return {"bytes": 12.0 * n + 3 * 1080 * 1080, "flops": 20.0 * n}
    out = {"log": 12.0 * n + 4 * E.E_COUNT * case["steps"], "grad": 200.0, "loss": 4.0}.get(kind, 12.0 * n)
    return {"bytes": 24.0 * n + out, "flops": (128.0 if kind == "grad" else 32.0) * pairs * case["steps"]}


# ------------------------------------------------------- FP64 restatement ---
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Box:
    """The system as flat FP64 tensors: compound particles compound by compound, then waters."""

    def __init__(self, system):
        dev, f8 = _dev(), torch.float64
        self.L, self.dt = float(np.float32(system.spec.box_len)), system.spec.dt
        pp = system.forcefield["particle_parameters"][0]
        c, s = system.compounds, system.solvents
        n_of = [int(k) for k in c["n_particles"]] if len(c) else []
        base = np.concatenate([[0], np.cumsum(n_of)]).astype(np.int64)
        self.n_of, self.base, self.n_cp, self.n_s = n_of, base, int(base[-1]), len(s)
        self.n = self.n_cp + self.n_s
        x = [system.states[k]["positions"][:m] for k, m in enumerate(n_of)] + [s["pos"]]
        p = [c[k]["prev_positions"][:m] for k, m in enumerate(n_of)] + [s["pos_tsub1"]]
        t = [c[k]["atom_types"][:m] for k, m in enumerate(n_of)] + [np.zeros(len(s), np.uint8)]
        self.x32 = torch.as_tensor(np.concatenate(x), device=dev)
        self.x = self.x32.to(f8)
        self.prev = torch.as_tensor(np.concatenate(p), device=dev).to(f8)
        self.v = (self.x - self.prev) / self.dt
        self.types = torch.as_tensor(np.concatenate(t).astype(np.int64), device=dev)
        self.n_types = int(self.types.max()) + 1
        par = lambda k: torch.as_tensor(pp[k][: self.n_types].astype(np.float64), device=dev)  # noqa: E731
        self.mass_t, self.sigma_t, self.eps_t = par("mass"), par("sigma"), par("epsilon")
        self.m = self.mass_t[self.types][:, None]
        excl, terms = set(), {"singlebonds": [], "anglebonds": [], "dihedrals": []}
        for k in range(len(n_of)):
            for q in range(n_of[k]):
                ig = c[k]["lj_ignore_list"][q]
                for z in range(int(ig["n_ignores"])):
                    excl.add((int(base[k]) + q) * self.n + int(base[ig["compound_ids"][z]]) + int(ig["local_ids"][z]))
            for kind, cnt in (("singlebonds", "n_singlebonds"), ("anglebonds", "n_anglebonds"),
                              ("dihedrals", "n_dihedrals")):
                for z in range(int(c[k][cnt])):
                    term = c[k][kind][z]
                    terms[kind].append(([int(base[k]) + int(a) for a in term["atom_indexes"]], term))
        for br in system.bridges:
            at = lambda a: int(base[br["particle_refs"][a]["compound_id"]]) + int(  # noqa: E731
                br["particle_refs"][a]["local_id_compound"])
            for kind, cnt in (("singlebonds", "n_singlebonds"), ("anglebonds", "n_anglebonds"),
                              ("dihedrals", "n_dihedrals")):
                for z in range(int(br[cnt])):
                    term = br[kind][z]
                    terms[kind].append(([at(int(a)) for a in term["atom_indexes"]], term))
        self.excl = torch.as_tensor(sorted(excl), dtype=torch.int64, device=dev)

        def flat(kind, width, *names):
            rows = terms[kind]
            ix = torch.as_tensor([r[0] for r in rows], dtype=torch.int64, device=dev).reshape(-1, width)
            return ix, [torch.as_tensor([float(r[1][k]) for r in rows], dtype=f8, device=dev) for k in names]

        self.bonds, (self.b0, self.kb) = flat("singlebonds", 2, "b0", "kb")
        self.angles, (self.t0, self.kt) = flat("anglebonds", 3, "theta_0", "k_theta")
        self.dihs, (self.p0, self.kp, self.nd) = flat("dihedrals", 4, "phi_0", "k_phi", "n")

    def image(self, d):
        return d - self.L * torch.round(d.detach() / self.L)

    def theta(self):
        """(sigma, epsilon, three scales, one constant pair per bonded kind: the boxes have one type of each)."""
        one = torch.ones(3, dtype=torch.float64, device=self.x.device)
        parts = [self.sigma_t, self.eps_t, one]
        for ix, c, k in ((self.bonds, self.b0, self.kb), (self.angles, self.t0, self.kt),
                         (self.dihs, self.p0, self.kp)):
            if len(ix):
                parts.append(torch.stack([c[0], k[0]]))
        return torch.cat(parts)

    def layout(self, flat):
        """A flat (n, 3) result as (compounds, 64, 3) and (waters, 3)."""
        a = np.zeros((len(self.n_of), 64, 3))
        h = flat.cpu().numpy()
        for k, m in enumerate(self.n_of):
            a[k, :m] = h[self.base[k]: self.base[k] + m]
        return [a, h[self.n_cp:].copy()]


def _pairs(b, x, radius):
    """All pairs i < j within radius (minimum image), bonded exclusions dropped."""
    x = torch.remainder(x.detach(), b.L)
    n, m = len(x), int(b.L / radius)
    got = []
    if m < 3:
        for lo in range(0, n, 1024):
            d = b.image(x[None, :, :] - x[lo: lo + 1024, None, :])
            i, j = torch.nonzero((d * d).sum(-1) < radius * radius, as_tuple=True)
            got.append(torch.stack([i + lo, j]))
    else:
        cell = torch.clamp((x * (m / b.L)).long(), max=m - 1)
        key = (cell[:, 0] * m + cell[:, 1]) * m + cell[:, 2]
        order = torch.argsort(key)
        count = torch.bincount(key, minlength=m ** 3)
        first = torch.cumsum(count, 0) - count
        width = int(count.max())
        slot = first[:, None] + torch.arange(width, device=x.device)[None, :]
        there = torch.arange(width, device=x.device)[None, :] < count[:, None]
        ids = torch.where(there, order[torch.clamp(slot, max=n - 1)], -1)
        xyz = torch.stack(torch.meshgrid(*[torch.arange(m, device=x.device)] * 3, indexing="ij"), -1).reshape(-1, 3)
        for off in range(27):
            o = torch.tensor([off // 9 - 1, off // 3 % 3 - 1, off % 3 - 1], device=x.device)
            nb = (xyz + o) % m
            nbk = (nb[:, 0] * m + nb[:, 1]) * m + nb[:, 2]
            for lo in range(0, m ** 3, 1024):
                a, c = ids[lo: lo + 1024], ids[nbk[lo: lo + 1024]]
                d = b.image(x[c.clamp(min=0)][:, None, :, :] - x[a.clamp(min=0)][:, :, None, :])
                ok = ((d * d).sum(-1) < radius * radius) & (a >= 0)[:, :, None] & (c >= 0)[:, None, :]
                z, p, q = torch.nonzero(ok, as_tuple=True)
                got.append(torch.stack([a[z, p], c[z, q]]))
    ij = torch.cat(got, 1)
    ij = ij[:, ij[0] < ij[1]]
    if len(b.excl):
        near = torch.nonzero(ij[1] < b.n_cp).reshape(-1)
        drop = near[torch.isin(ij[0, near] * b.n + ij[1, near], b.excl)]
        keep = torch.ones(ij.shape[1], dtype=torch.bool, device=x.device)
        keep[drop] = False
        ij = ij[:, keep]
    return ij


def _terms(b, x, ij, rc, theta=None, stretch=1.0, hist=None):
    """Energies (LJ, bond, angle, dihedral) at x; stretch scales every distance (the virial's derivative);
    hist = (bins, r_max): the RDF-bin occupancies too."""
    nt = b.n_types
    sig, eps = (b.sigma_t, b.eps_t) if theta is None else (theta[:nt], theta[nt: 2 * nt])
    scale = [1.0, 1.0, 1.0] if theta is None else theta[2 * nt: 2 * nt + 3]
    par, at = [], 2 * nt + 3
    for ix, c, k in ((b.bonds, b.b0, b.kb), (b.angles, b.t0, b.kt), (b.dihs, b.p0, b.kp)):
        if theta is None or not len(ix):
            par.append((c, k))
        else:
            par.append((theta[at], theta[at + 1]))
            at += 2
    d = b.image(x[ij[1]] - x[ij[0]]) * stretch
    r2 = (d * d).sum(-1)
    ti, tj = b.types[ij[0]], b.types[ij[1]]
    s2 = (0.5 * (sig[ti] + sig[tj])) ** 2 / r2
    s6 = s2 ** 3
    t = torch.clamp((rc * rc - r2) / (rc * rc - (rc - 0.2) ** 2), 0.0, 1.0)
    lj = 4.0 * torch.sqrt(eps[ti] * eps[tj]) * (s6 * s6 - s6) * t ** 3 * (10.0 + t * (-15.0 + 6.0 * t))
    zero = lj.sum() * 0.0
    e = [lj.sum(), zero, zero, zero]
    vec = lambda i, j: b.image(x[j] - x[i]) * stretch  # noqa: E731
    if len(b.bonds):
        r = vec(b.bonds[:, 0], b.bonds[:, 1]).norm(dim=-1)
        e[1] = (0.5 * scale[0] * par[0][1] * (r - par[0][0]) ** 2).sum()
    if len(b.angles):
        u, v = vec(b.angles[:, 1], b.angles[:, 0]), vec(b.angles[:, 1], b.angles[:, 2])
        th = torch.atan2(torch.linalg.cross(u, v).norm(dim=-1), (u * v).sum(-1))
        e[2] = (0.5 * scale[1] * par[1][1] * (th - par[1][0]) ** 2).sum()
    if len(b.dihs):
        b1, b2, b3 = (vec(b.dihs[:, k], b.dihs[:, k + 1]) for k in range(3))
        m1, m2 = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
        phi = torch.atan2(b2.norm(dim=-1) * (b1 * m2).sum(-1), (m1 * m2).sum(-1))
        e[3] = (scale[2] * par[2][1] * (1.0 + torch.cos(b.nd * phi - par[2][0]))).sum()
    if hist is None:
        return e
    bins, dr = hist[0], hist[1] / hist[0]
    near = torch.nonzero(r2.detach() < (hist[1] + dr) ** 2).reshape(-1)
    u = torch.sqrt(r2[near]) / dr
    b0 = torch.floor(u.detach() - 0.5).long() - 1
    h = torch.zeros(bins + 8, dtype=x.dtype, device=x.device)
    for k in range(4):
        w = torch.abs(u - (b0 + k) - 0.5)
        spline = torch.where(w < 0.5, 0.75 - w * w, torch.where(w < 1.5, 0.5 * (1.5 - w) ** 2, torch.zeros_like(w)))
        h = h.index_add(0, torch.clamp(b0 + k, -4, bins + 3) + 4, spline)
    return e, h[4: 4 + bins] / b.n


class _List:
    """Pairs within the cutoff plus a margin, found again when a particle has used it up."""

    def __init__(self, b, rc, margin=0.12):
        self.b, self.rc, self.margin, self.at, self.made = b, rc, margin, None, []

    def of(self, x):
        x = x.detach()
        if self.at is None or float((x - self.at).norm(dim=-1).max()) > 0.49 * self.margin:
            self.at = x.clone()
            if self.b.L < 2 * (self.rc + self.margin):
                self.margin = 0.5 * self.b.L - self.rc - 1e-6
            self.made.append(_pairs(self.b, x, self.rc + self.margin))
        return len(self.made) - 1


def _forces(b, x, ij, rc, virial=False):
    x = x.detach().requires_grad_(True)
    s = torch.ones((), dtype=x.dtype, device=x.device, requires_grad=True)
    e = _terms(b, x, ij, rc, stretch=s if virial else 1.0)
    wrt = (x, s) if virial else (x,)
    g = torch.autograd.grad(sum(e), wrt)
    return -g[0], [float(v.detach()) for v in e] + [-float(g[1]) if virial else 0.0]


def _kinetic(b, v):
    ke = float((0.5 * b.m * v * v).sum())
    return ke, 2.0 * ke / (3.0 * b.n * R_GAS)


def _row(e, ke, temp):
    """energies in the order of engine.E_*"""
    return [e[0], e[1], e[2], e[3], ke, e[4], temp, sum(e[:4]) + ke]


def _dynamics(case, b):
    """The kick-drift velocity Verlet of the physics path; positions after the steps, energies of each."""
    nl, x, v, rows, before = _List(b, case["cutoff"]), b.x, b.v, [], None
    for _ in range(case["steps"]):
        k = nl.of(x)
        nl.made = [None] * k + nl.made[k:]
        f, e = _forces(b, x, nl.made[k], case["cutoff"], virial=case["kind"] == "log")
        full = v + f / b.m * (0.5 * b.dt)
        lam = 1.0
        if case["thermostat"] == "berendsen" or case["kind"] == "log":
            ke, temp = _kinetic(b, full)
            if case["thermostat"] == "berendsen" and before is not None:
                lam = math.sqrt(1.0 + b.dt / 1e-4 * (300.0 / before - 1.0))
            before = temp
            rows.append(_row(e, ke, temp))
        v = lam * full + f / b.m * (0.5 * b.dt)
        x = x + v * b.dt
    return x, rows


def _trajectory(case, b, spec, want_grad):
    """Loss of the unrolled constant-energy steps and, by the adjoint of each step, its gradient."""
    rc, T, hist = case["cutoff"], spec["n_steps"], (spec["n_bins"], spec["r_max"])
    target = torch.as_tensor(spec["target"], device=b.x.device)
    theta = b.theta()
    nl, x, v, xs, ks, total = _List(b, rc, 0.2), b.x, b.v, [b.x], [], 0.0

    def state_loss(y, ij, th):
        e, h = _terms(b, y, ij, rc, th, hist=hist)
        return (spec["w_energy"] * sum(e) / b.n + spec["w_rdf"] * ((h - target) ** 2).sum()) / T

    for _ in range(T):
        ks.append(nl.of(x))
        f, _e = _forces(b, x, nl.made[ks[-1]], rc)
        v = v + f / b.m * b.dt
        x = x + v * b.dt
        xs.append(x)
    ks.append(nl.of(x))
    g, lx, lv = torch.zeros_like(theta), torch.zeros_like(x), torch.zeros_like(x)
    for n in range(T, 0, -1):
        if want_grad:
            y, th = xs[n].detach().requires_grad_(True), theta.detach().requires_grad_(True)
            l = state_loss(y, nl.made[ks[n]], th)
            gx, gt = torch.autograd.grad(l, (y, th))
            lx, g = lx + gx, g + gt
            lv = lv + b.dt * lx
            y, th = xs[n - 1].detach().requires_grad_(True), theta.detach().requires_grad_(True)
            e = sum(_terms(b, y, nl.made[ks[n - 1]], rc, th))
            force = -torch.autograd.grad(e, y, create_graph=True)[0]
            gx, gt = torch.autograd.grad((force * (lv * b.dt / b.m)).sum(), (y, th))
            lx, g = lx + gx, g + gt
        else:
            with torch.no_grad():
                l = state_loss(xs[n], nl.made[ks[n]], theta)
        total += float(l.detach())
    return total, g


def _reference(case, b, system):
    """The reference's step in FP64 (lists by its own FP32 test): bonded forms, no LJ cutoff inside its lists,
    Stormer-Verlet, the 40-step thermostat."""
    C, Lf, dev = np.float32(case["cutoff"]) / np.float32(2.0), np.float32(b.L), b.x.device
    nc, unit = len(b.n_of), lambda a: a / a.norm(dim=-1, keepdim=True).clamp(min=1e-300)  # noqa: E731

    def distance32(a, c):
        d = c - a
        half = float(Lf / np.float32(2.0))
        c = torch.where(-d > half, c + float(Lf), c)
        c = torch.where((a - c) < -half, c - float(Lf), c)
        d = a - c
        return torch.sqrt(d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2])

    comp = [slice(int(b.base[k]), int(b.base[k + 1])) for k in range(nc)]
    sol = slice(b.n_cp, b.n)
    w32 = b.x32[sol]
    key = [b.x32[int(b.base[k]) + int(system.compounds[k]["key_particle_index"])] for k in range(nc)]
    ball = [system.compounds[k]["confining_particle_sphere"] for k in range(nc)]
    near = [distance32(key[k], w32) < float(C + (ball[k] + C)) for k in range(nc)]
    touch = [[j for j in range(nc) if j != i and bool(
        distance32(key[min(i, j)], key[max(i, j)]) < float(C + ((ball[min(i, j)] + ball[min(i, j)]) + C)))]
        for i in range(nc)]
    ww = _pairs(b, b.x, 2.0 * float(C) + 1e-4)
    ww = ww[:, ww[0] >= b.n_cp]
    ww = ww[:, distance32(b.x32[ww[0]], b.x32[ww[1]]) < float(C + C)]
    allowed = {}
    for i in range(nc):
        for j in [i] + touch[i]:
            p = torch.arange(comp[i].start, comp[i].stop, device=dev)
            q = torch.arange(comp[j].start, comp[j].stop, device=dev)
            m = ~torch.isin(p[:, None] * b.n + q[None, :], b.excl)
            allowed[i, j] = m & (p[:, None] != q[None, :])
    sig, eps = b.sigma_t[b.types], b.eps_t[b.types]

    def lj(d, s, e):
        d2 = (d * d).sum(-1)
        q = (s * s / d2) ** 3
        return d * (24.0 * e * q / d2 * (1.0 - 2.0 * q))[..., None]

    def to_image(x, at):
        return x + b.L * torch.round((at - x) / b.L)

    def forces(x):
        f = torch.zeros_like(x)
        if len(b.bonds):
            d = x[b.bonds[:, 0]] - x[b.bonds[:, 1]]
            fr = unit(d) * (-b.kb * (d.norm(dim=-1) - b.b0))[:, None]
            f.index_add_(0, b.bonds[:, 0], fr).index_add_(0, b.bonds[:, 1], -fr)
        if len(b.angles):
            p, q, r = (x[b.angles[:, k]] for k in range(3))
            u, w = p - q, r - q
            ang = torch.atan2(torch.linalg.cross(u, w).norm(dim=-1), (u * w).sum(-1))
            k = (b.kt * (ang - b.t0))[:, None]
            fu = unit(torch.linalg.cross(u, torch.linalg.cross(w, u))) * k
            fw = unit(torch.linalg.cross(w, torch.linalg.cross(u, w))) * k
            f.index_add_(0, b.angles[:, 0], fu).index_add_(0, b.angles[:, 2], fw)
            f.index_add_(0, b.angles[:, 1], -(fu + fw))
        if len(b.dihs):
            l, lm, rm, r = (x[b.dihs[:, k]] for k in range(4))
            n1 = unit(torch.linalg.cross(l - lm, rm - lm))
            n2 = unit(torch.linalg.cross(lm - rm, r - rm))
            tor = torch.atan2(torch.linalg.cross(n1, n2).norm(dim=-1), (n1 * n2).sum(-1))
            flip = ((l + n1 - r).norm(dim=-1) < (l - n1 - r).norm(dim=-1))[:, None]
            n1, n2 = torch.where(flip, n1, -n1), torch.where(flip, -n2, n2)
            k = (b.kp * torch.sin(b.nd * tor - b.p0))[:, None]
            f.index_add_(0, b.dihs[:, 0], n1 * k).index_add_(0, b.dihs[:, 3], n2 * k)
            mid = -0.5 * (n1 + n2) * k
            f.index_add_(0, b.dihs[:, 1], mid).index_add_(0, b.dihs[:, 2], mid)
        w = x[sol]
        for k in range(nc):
            p = x[comp[k]]
            im = to_image(w, p[0])
            d = p[None, :, :] - im[:, None, :]
            s = 0.5 * (sig[comp[k]] + b.sigma_t[0])[None, :]
            # waters feel every compound with the arithmetic epsilon, compounds their listed waters with the geometric
            f[sol] += lj(d, s, 0.5 * (eps[comp[k]] + b.eps_t[0])[None, :]).sum(1)
            back = lj(-d, s, torch.sqrt(eps[comp[k]] * b.eps_t[0])[None, :])
            f[comp[k]] += (back * near[k][:, None, None]).sum(0)
            for j in [k] + touch[k]:
                o = x[comp[j]] if j == k else to_image(x[comp[j]], p[0])
                mix = torch.sqrt(eps[comp[k]][:, None] * eps[comp[j]][None, :]) if j == k else 0.5 * (
                    eps[comp[k]][:, None] + eps[comp[j]][None, :])
                ok = allowed[k, j]
                dd = torch.where(ok[..., None], o[None, :, :] - p[:, None, :], torch.ones_like(p[0]))
                s2 = 0.5 * (sig[comp[k]][:, None] + sig[comp[j]][None, :])
                f[comp[k]] += (lj(dd, s2, mix) * ok[..., None]).sum(1)
        pw = lj(b.image(x[ww[1]] - x[ww[0]]), b.sigma_t[0], b.eps_t[0])
        return f.index_add_(0, ww[0], pw).index_add_(0, ww[1], -pw)

    x, prev, lam, snap = b.x, b.prev, 1.0, None
    for step in range(1, case["steps"] + 1):
        new = 2.0 * x - prev + forces(x) * (b.dt / b.m * b.dt)
        prev, x = x, x + (new - x) * lam
        lam = 1.0
        if step % 40 == 38:
            snap = x
        if step % 40 == 0:
            speed = (x - snap).norm(dim=-1, keepdim=True) * 0.5 / b.dt
            temp = float((0.5 * b.m * speed * speed).mean()) * 2.0 / (3.0 * 8.3145)
            lam = min(max(300.0 / temp, 0.9), 1.1)
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "render":
        return None          # a picture is bytes
    system = _system(case, seed)
    b = _Box(system)
    if kind == "evaluate":
        f, e = _forces(b, b.x, _pairs(b, b.x, case["cutoff"]), case["cutoff"], virial=True)
        ke, temp = _kinetic(b, b.v + f / b.m * (0.5 * b.dt))
        return b.layout(f) + [np.array(_row(e, ke, temp))]
    if kind in ("grad", "loss"):
        loss, g = _trajectory(case, b, _loss_spec(case), kind == "grad")
        loss = torch.tensor(loss, dtype=torch.float64)
        return [loss, g.cpu()] if kind == "grad" else [loss]
    if kind == "reference":
        if case["steps"] > 200 or (system.bridges is not None and len(system.bridges)):
            return None      # its lists change after 200 steps
        return b.layout(_reference(case, b, system))
    x, rows = _dynamics(case, b)
    out = b.layout(x)
    return out + [np.array(rows)] if kind == "log" else out
