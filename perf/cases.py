"""Measured cases of the gravity step and the Fourier work around it.

Every case is a call sequence a program makes through the package's public entry points:

* ``step``       tree build, kick and drift of one box, all particles active.  The program holds
                 its particles in device arrays of its own: a pass hands them over
                 (``upload_device``), steps, and takes the new state back (``download_device``).
* ``substep``    one level of the multistep ladder: the rung partition, the tree over the active
                 particles, their kick (both half kicks, rungs assigned) and the drift of the
                 level.  (``step_hierarchical`` makes the same calls level by level; the rungs it
                 assigns on the way decide the order of the particles it returns, so that a
                 particle on a rung boundary would reorder its whole output.)
* ``ensemble``   the step of many independent boxes of uneven sizes in one set of launches.
* ``lightcone``  a drift with the lightcone capture, the entries handed over and counted on the
                 HEALPix map they belong to (their order is unspecified).
* ``initialize`` Zel'dovich or 2LPT initial conditions from a power table.
* ``power``      the power spectrum of the particles.

Boxes are synthetic, made on the GPU from the seed, with the shapes of the benchmark's
configurations: a Zel'dovich-displaced lattice, and the clustered mix of 70% lattice and 30%
Plummer spheres.  Unless a case is ``fresh`` (particles as their generator ordered them, the
first step of a run or of a request), they come as a previous step left them: in the tree's
order, kicked and drifted.
"""
import math

import numpy as np
import torch

import cosmictiger_b200 as ct
from cosmictiger_b200 import ics

SELF_PHI = 693.0 / 256.0
COSMO = dict(omega_m=0.3111, z0=49.0, hubble=0.6732, sigma8=0.8607, H0=1.0)
IC_BOX = 500.0  # Mpc


# ------------------------------------------------------------------------------------- cases
def _step(n, box, theta, order=7, fresh=False, save_force=True, do_phi=True, bucket=128):
    return dict(kind="step", n=n, box=box, theta=theta, order=order, fresh=fresh, save_force=save_force, do_phi=do_phi, bucket=bucket)


def listed():
    return [
        # the smallest box of the ensembles on its own: launches and host round trips
        dict(_step(16 ** 3, "lattice", 0.7), name="step_16"),
        # the plain single-box configuration
        dict(_step(64 ** 3, "lattice", 0.7), name="step_64"),
        # a count that is no cube, the low expansion order, no potential, first step of a run
        dict(_step(1000003, "clustered", 0.7, order=5, fresh=True, do_phi=False), name="step_1m_order5"),
        # the benchmark's box, all particles active
        dict(_step(256 ** 3, "clustered", 0.55, save_force=False), name="step_256"),
        # a fine level of a small box's ladder: few active particles
        dict(kind="substep", n=64 ** 3, box="clustered", theta=0.55, active=0.1, level=2, name="substep_64"),
        # a level of the benchmark box's ladder
        dict(kind="substep", n=256 ** 3, box="clustered", theta=0.55, active=0.3, level=1, name="substep_256"),
        # many small requests batched
        dict(kind="ensemble", nbox=64, nmin=16, nmax=64, theta=0.55, fresh=True, name="ensemble_64"),
        # the batched ensemble, a quarter of its 512 boxes
        dict(kind="ensemble", nbox=128, nmin=16, nmax=128, theta=0.55, fresh=False, name="ensemble_128"),
        # a drift of a run that keeps a lightcone
        dict(kind="lightcone", n=128 ** 3, nside=64, name="lightcone_128"),
        # initial conditions of a small and of the benchmark's size
        dict(kind="initialize", grid=64, twolpt=False, name="zeldovich_64"),
        dict(kind="initialize", grid=256, twolpt=True, name="2lpt_256"),
        # the spectrum of the benchmark's box
        dict(kind="power", n=256 ** 3, grid=256, fold=1, name="power_256"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step"] * 4 + ["substep"] * 2 + ["ensemble"] * 2 + ["initialize"] * 2 + ["power"] * 2 + ["lightcone"])
    if kind == "step":
        return _step(int(_log(rng, 16 ** 3, 256 ** 3)), rng.choice(["lattice", "clustered"]), round(rng.uniform(0.4, 0.75), 3),
                     order=rng.choice([7, 7, 5]), fresh=rng.random() < 0.3, save_force=rng.random() < 0.5, do_phi=rng.random() < 0.6,
                     bucket=rng.choice([128, 128, 64, 96]))
    if kind == "substep":
        return dict(kind=kind, n=int(_log(rng, 32 ** 3, 256 ** 3)), box="clustered", theta=round(rng.uniform(0.45, 0.7), 3),
                    active=round(_log(rng, 0.02, 0.6), 3), level=rng.choice([1, 2, 3]))
    if kind == "ensemble":
        nmin = rng.choice([16, 20, 32])
        return dict(kind=kind, nbox=int(_log(rng, 3, 100)), nmin=nmin, nmax=rng.randrange(nmin + 8, 129), theta=round(rng.uniform(0.5, 0.7), 3),
                    fresh=rng.random() < 0.5)
    if kind == "initialize":
        return dict(kind=kind, grid=2 * int(_log(rng, 16, 128)), twolpt=rng.random() < 0.5)
    if kind == "power":
        return dict(kind=kind, n=int(_log(rng, 32 ** 3, 256 ** 3)), grid=2 * int(_log(rng, 16, 128)), fold=rng.choice([1, 1, 2, 4]))
    return dict(kind=kind, n=int(_log(rng, 32 ** 3, 200 ** 3)), nside=rng.choice([16, 64, 256]))


# ------------------------------------------------------------------------------------ inputs
def _displacements(n, index, rms, gen, count):
    """`count` of the n^3 lattice points (3, count) with a Zel'dovich displacement of RMS `rms`
    mean spacings, P(k) ~ k^index cut at the lattice's Nyquist wavenumber."""
    k1 = torch.fft.fftfreq(n, 1.0 / n, device=gen.device)
    kz = torch.fft.rfftfreq(n, 1.0 / n, device=gen.device)
    k2 = (k1 ** 2)[:, None, None] + (k1 ** 2)[None, :, None] + (kz ** 2)[None, None, :]
    amp = torch.where((k2 > 0) & (k2 < (n / 2) ** 2), k2.clamp(min=1.0) ** (index / 4.0 - 1.0), torch.zeros_like(k2))
    del k2
    delta = torch.complex(torch.randn(amp.shape, generator=gen, device=gen.device), torch.randn(amp.shape, generator=gen, device=gen.device)) * amp
    del amp
    keep = None if count == n ** 3 else torch.randperm(n ** 3, generator=gen, device=gen.device)[:count].sort().values
    psi = torch.empty((3, count), device=gen.device)
    for d, K in enumerate((k1[:, None, None], k1[None, :, None], kz[None, None, :])):
        f = torch.fft.irfftn(1j * K * delta, s=(n, n, n)).reshape(-1)
        psi[d] = f if keep is None else f[keep]
    psi *= rms / n / psi.square().sum(0).mean().sqrt()
    at = torch.arange(n ** 3, device=gen.device) if keep is None else keep
    base = torch.stack([at // (n * n), at // n % n, at % n]).double() / n
    return base + psi, psi


def _plummer(count, nspheres, gen):
    """`count` positions in Plummer spheres: masses dN/dM ~ M^-1.9 over 10^2..10^5, scale radii
    0.002 (M / 10^3)^(1/3), cut at ten of them."""
    dev = gen.device
    u = torch.rand(nspheres, generator=gen, device=dev, dtype=torch.float64)
    m = (1e2 ** -0.9 + u * (1e5 ** -0.9 - 1e2 ** -0.9)) ** (-1.0 / 0.9)
    owner = torch.searchsorted(m.cumsum(0) / m.sum(), torch.rand(count, generator=gen, device=dev, dtype=torch.float64).sort().values).clamp(max=nspheres - 1)
    centre = torch.rand((3, nspheres), generator=gen, device=dev, dtype=torch.float64)
    a = 0.002 * (m / 1e3) ** (1.0 / 3.0)
    U = torch.rand(count, generator=gen, device=dev, dtype=torch.float64).clamp(min=1e-12) * (1000.0 / 101.0 ** 1.5)
    r = a[owner] / (U ** (-2.0 / 3.0) - 1.0).sqrt()
    way = torch.randn((3, count), generator=gen, device=dev, dtype=torch.float64)
    return centre[:, owner] + way * (r / way.square().sum(0).sqrt())


def _fixed32(p):
    """Positions as 32-bit fixed point (3, n), held as int32 bits."""
    return ((p - p.floor()) * 4294967296.0).to(torch.int64).to(torch.int32)


def _particles(n, box, gen, index=None, rms=None):
    """(positions int32 bits (3, n), velocities (n, 3)) of a lattice or clustered box."""
    nl = n if box == "lattice" else int(round(0.7 * n))
    side = max(2, round(n ** (1.0 / 3.0)))
    side += side ** 3 < nl
    index = index if index is not None else (-2.0 if box == "lattice" else -1.5)
    rms = rms if rms is not None else (0.25 if box == "lattice" else 0.5)
    p, v = _displacements(side, index, rms, gen, nl)
    x = torch.zeros((3, n), dtype=torch.int32, device=gen.device)
    vel = torch.zeros((n, 3), dtype=torch.float32, device=gen.device)
    x[:, :nl] = _fixed32(p)
    vel[:nl] = v.t()
    if n > nl:
        x[:, nl:] = _fixed32(_plummer(n - nl, max(1, round(20000 * n / 256 ** 3)), gen))
    return x, vel


def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


class State:
    """The particles in the program's own device arrays, the library's context and box, and the
    arrays that take the results."""

    def __init__(self, case, n, order=7, counts=None):
        self.case, self.n = case, n
        self.ctx = ct.Context(order=order)
        self.box = self.ctx.box(n) if counts is None else self.ctx.ensemble(counts)
        self.stream = torch.cuda.ExternalStream(self.ctx.stream_handle())
        self.x = torch.empty((3, n), dtype=torch.int32, device="cuda")
        self.v = torch.empty((n, 3), dtype=torch.float32, device="cuda")
        self.r = torch.zeros(n, dtype=torch.int8, device="cuda")
        self.out_x, self.out_v, self.out_r = torch.empty_like(self.x), torch.empty_like(self.v), torch.empty_like(self.r)
        self.out_g = None
        self.unit = torch.tensor(1.0 / 4294967296.0, dtype=torch.float64)

    def wait(self):
        """The library's stream after what torch was given so far."""
        self.stream.wait_stream(torch.cuda.current_stream())

    def upload(self):
        x = self.x
        self.box.upload_device(x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(), self.v.data_ptr(), self.r.data_ptr())

    def download(self, forces=False, to=None):
        x, v, r = to or (self.out_x, self.out_v, self.out_r)
        g = [None] * 4
        if forces:
            if self.out_g is None:
                self.out_g = torch.empty((4, self.n), device="cuda")
            g = [q.data_ptr() for q in self.out_g]
        self.box.download_device(x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(), v.data_ptr(), r.data_ptr(), *g)

    def outputs(self, forces=False, phi=False):
        """Positions as box units in [-0.5, 0.5), velocities, rungs (and forces, potential)."""
        out = {"pos": self.out_x * self.unit, "vel": self.out_v, "rung": self.out_r}
        if forces:
            out["force"] = self.out_g[:3]
            if phi:
                out["pot"] = self.out_g[3]
        return out


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    if kind == "initialize":
        s = State(case, case["grid"] ** 3)
        s.table = _table(case, seed)
        return s
    if kind == "ensemble":
        # the boxes' sizes and spectra: n log-uniform, index -2.5..-1, RMS displacement 0.1..0.6
        rng = np.random.default_rng(7919)  # sizes belong to the case, so that work does not change with the seed
        ns = np.rint(np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]), case["nbox"]))).astype(int)
        ns[0] = case["nmax"]
        index, rms = rng.uniform(-2.5, -1.0, case["nbox"]), rng.uniform(0.1, 0.6, case["nbox"])
        counts = [int(n) ** 3 for n in ns]
        s = State(case, sum(counts), counts=counts)
        at = 0
        for n, i, q in zip(counts, index, rms):
            s.x[:, at:at + n], s.v[at:at + n] = _particles(n, "lattice", gen, float(i), float(q))
            at += n
        h = np.array([ics.softening(n, 0.02) for n in counts])
        s.box.set_box_params(h, np.array([1.0 / n for n in counts]))
        s.h, s.GM = float(h.max()), 1.0
        s.own_h = torch.repeat_interleave(torch.from_numpy(h), torch.tensor(counts)).cuda()
    else:
        s = State(case, case["n"], order=case.get("order", 7))
        s.x[:], s.v[:] = _particles(case["n"], case.get("box", "clustered"), gen)
        s.h, s.GM = ics.softening(case["n"], 0.02), 1.0 / case["n"]
        s.own_h = s.h
    s.wait()
    if kind == "substep":
        _assign_rungs(s)
    elif kind in ("step", "ensemble"):
        # the step that all but a hundredth of the particles can take
        dt = _own_steps(s, to=(s.out_x, s.out_v, s.out_r))
        s.t0 = float(dt.kthvalue(max(1, s.n // 100)).values)
        if not case["fresh"]:
            s.upload()
            _gravity_step(s)
            s.download(to=(s.x, s.v, s.r))
    elif kind == "power":
        s.upload()  # the spectrum is taken of a resident box
    return s


def _own_steps(s, to):
    """Every particle's own time step by the rung rule, eta sqrt(h / |g|), in the tree's order;
    the particles themselves, in that order, go to `to`."""
    c, b = s.case, s.box
    s.upload()
    b.tree_create(c["theta"], s.h, c.get("bucket", 128))
    kp = ct.KickParams.make(theta=c["theta"], h=s.h, GM=s.GM, eta=ics.eta_default(), t0=1.0, ascending=False, descending=False)
    if c["kind"] == "ensemble":
        b.kick_ensemble(kp)
    else:
        b.kick(kp)
    s.download(forces=True, to=to)
    dt = ics.eta_default() * (s.own_h / s.out_g[:3].double().square().sum(0).sqrt().clamp(min=1e-30)).sqrt()
    s.out_g = None
    return dt


def _assign_rungs(s):
    """The state in which a ladder visits a level above its base: all particles in the base
    level's tree order, rungs from the rung rule with the top step set so that the wanted share
    is on the level or above."""
    c = s.case
    dt = _own_steps(s, to=(s.x, s.v, s.r))
    s.t0 = float(dt.kthvalue(max(1, int(c["active"] * s.n))).values) * 2.0 ** (c["level"] - 1)
    s.r.copy_(torch.ceil(torch.log2(s.t0 / dt)).clamp(0, c["level"] + 1).to(torch.int8))
    s.wait()


def _table(case, seed):
    """A power.init-style table that covers the grid's wavenumbers, another slope for every seed, its
    power far below the grid scale (the rows of the field's Nyquist plane are drawn one by one and
    not Hermitian, so that a transform's result from it is its own)."""
    n = case["grid"]
    return ics.power_law_table(index=-1.5 - 0.3 * (seed % 1009) / 1009.0, kcut=0.15 * np.pi * n / IC_BOX / COSMO["hubble"])


# -------------------------------------------------------------------------------------- pass
def _gravity_step(s):
    c, b = s.case, s.box
    b.tree_create(c["theta"], s.h, c.get("bucket", 128))
    kp = ct.KickParams.make(theta=c["theta"], h=s.h, GM=s.GM, eta=ics.eta_default(), t0=s.t0, first_call=False, save_force=c.get("save_force", False),
                            do_phi=c.get("do_phi", True))
    kr = b.kick_ensemble(kp) if c["kind"] == "ensemble" else [b.kick(kp)]
    b.drift(0, 1.0, s.t0)
    return kr


def _returns(kr, phi=True):
    """What a run's log keeps of the kick returns."""
    e = [[k.kin, k.dkin] + [k.pot] * phi for k in kr]
    p = [[k.xmom, k.ymom, k.zmom, k.nmom] for k in kr]
    return {"max_rung": np.array([k.max_rung for k in kr]), "energy": np.array(e), "momentum": np.array(p)}


def run(s):
    c, b = s.case, s.box
    kind = c["kind"]
    if kind == "initialize":
        s.wait()
        r = b.initialize(c["grid"], IC_BOX, s.table[0], s.table[1], twolpt=c["twolpt"], **COSMO)
        s.download()
        out = s.outputs()
        out["dxmax"] = np.array(r["dxmax"] + (r["dxmax2"] if c["twolpt"] else []))
        return out
    if kind == "power":
        k, P, e = b.power_spectrum(c["grid"], IC_BOX, c["fold"])
        return {"k": k, "P": P, "err": e}
    s.wait()
    s.upload()
    if kind == "lightcone":
        dt = 0.005
        b.drift_lightcone(0, 1.0, dt, 0.7, 0.7 + dt, 1.6, c["nside"])
        entries = b.lightcone()
        s.download()
        return {"map": np.bincount(entries["pix"], minlength=12 * c["nside"] ** 2), "x": s.out_x, "vel": s.out_v}
    if kind == "substep":
        b.sort_by_rung(0)
        first = b.sort_by_rung(c["level"])
        b.tree_create(c["theta"], s.h, 128, min_rung=c["level"])
        kr = b.kick(ct.KickParams.make(theta=c["theta"], h=s.h, GM=s.GM, eta=ics.eta_default(), min_rung=c["level"], t0=s.t0, save_force=False,
                                       first_call=False, top=False, do_phi=False))
        b.drift(c["level"], 1.0, s.t0 / 2 ** c["level"])
        s.download()
        return dict(s.outputs(), first=first, **_returns([kr], phi=False))
    kr = _gravity_step(s)
    forces = c.get("save_force", False)
    s.download(forces)
    phi = c.get("do_phi", True)
    return dict(s.outputs(forces, phi), **_returns(kr, phi))


# -------------------------------------------------------------------------------------- work
def _counts(case):
    rng = np.random.default_rng(7919)
    ns = np.rint(np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]), case["nbox"]))).astype(int)
    ns[0] = case["nmax"]
    return [int(n) ** 3 for n in ns]


def _flops(case, n, nbox=1):
    """Interaction arithmetic of a kick of n active particles, by the reference's counts per
    interaction (within a fifth of the library's own counters at the listed sizes): a share for
    every particle, and the Ewald part of every box's coarsest nodes."""
    return n * 1.3e5 * (0.55 / case["theta"]) ** 2 * (0.8 if case.get("order", 7) == 5 else 1.0) + nbox * 3.7e9 * (0.7 / case["theta"]) ** 6


def work(case):
    kind = case["kind"]
    if kind == "initialize":
        n, fields = case["grid"] ** 3, 12 + 3 if case["twolpt"] else 3
        # written: positions, velocities, rungs; one inverse transform a field
        return {"bytes": 25.0 * n, "flops": fields * 2.5 * n * math.log2(n)}
    if kind == "power":
        g = case["grid"] ** 3
        return {"bytes": 12.0 * case["n"], "flops": 216.0 * 2 * case["n"] + 2.5 * g * math.log2(g)}
    if kind == "lightcone":
        return {"bytes": 2 * 25.0 * case["n"], "flops": 60.0 * case["n"]}
    if kind == "substep":
        return {"bytes": 2 * 25.0 * case["n"], "flops": _flops(case, 0.5 * case["active"] * case["n"])}  # (a sparser set of sources)
    n = sum(_counts(case)) if kind == "ensemble" else case["n"]
    return {"bytes": (50.0 + 16.0 * case.get("save_force", False)) * n, "flops": _flops(case, n, case.get("nbox", 1))}


def tolerance(case):
    kind = case["kind"]
    if kind == "lightcone":
        return "exact"
    if kind == "initialize":
        return {"rel": 6e-6, "max": 3e-4}  # 1.5e-6 from 64 bits
    if kind == "power":
        return {"rel": 2e-5, "max": 1e-3}  # single-precision deposits: 6.7e-6 from 64 bits
    # single-precision sums of forces that nearly cancel (potentials move by 1.4e-6, forces by 6e-7
    # with the particle-particle sums in another order); a particle on a rung boundary may fall to
    # either side, and its drift with it
    return {"rel": 6e-6, "max": 2e-3, "differ": 1e-3}


# -------------------------------------------------------------------- the results in 64 bits
EXACT_PARTICLES = 16384


def exact(case, seed):
    kind = case["kind"]
    if kind == "initialize":
        return _exact_initialize(case, seed)
    if kind == "power":
        return _exact_power(case, seed)
    if kind == "step" and case["n"] <= EXACT_PARTICLES:
        return _exact_step(case, seed)
    return None


def _tree_order(x, theta, hsoft, bucket):
    """Positions of the particles after the tree build's in-place partitions: a node splits at the
    midpoint of its longest side while it holds more than a bucket or is too large, the k-th
    particle of the upper half in its lower range changing places with the k-th of the lower
    half, from the right, in its upper range."""
    order = np.arange(x.shape[1])
    todo = [(0, x.shape[1], np.zeros(3), np.ones(3))]
    while todo:
        b, e, lo, hi = todo.pop()
        r = math.sqrt(float((0.25 * (hi - lo) ** 2).sum()))
        small = r < 0.25 * theta / (1.0 + theta) and r < 0.125 - 0.25 * hsoft
        if e - b <= bucket and (small or e == b):
            continue
        d = int(np.argmax(hi - lo))
        mid = 0.5 * (lo[d] + hi[d])
        low = x[d, order[b:e]] < mid * 4294967296.0
        m = int(low.sum())
        left = np.flatnonzero(~low[:m]) + b
        right = (np.flatnonzero(low[m:]) + b + m)[::-1]
        order[left], order[right] = order[right], order[left].copy()
        up, down = hi.copy(), lo.copy()
        up[d] = down[d] = mid
        todo += [(b, b + m, lo, up), (b + m, e, down, hi)]
    return order


def _exact_gravity(x, h, GM):
    """Force and potential (4, n) of a periodic box by a direct Ewald sum: nearest images softened
    inside h, splitting parameter 4."""
    dev, n, alpha = x.device, x.shape[1], 4.0
    out = torch.zeros((4, n), dtype=torch.float64, device=dev)
    p = x.double() / 4294967296.0
    reach = 1.5
    images = [(i, j, k) for i in range(-2, 3) for j in range(-2, 3) for k in range(-2, 3)
              if sum(max(abs(q) - 0.5, 0.0) ** 2 for q in (i, j, k)) < reach ** 2]
    step = max(1, 2 ** 24 // n)
    for a in range(0, n, step):
        xi = x[:, a:a + step]
        d = torch.stack([(xi[q][:, None] - x[q][None, :]).double() / 4294967296.0 for q in range(3)])  # wraps to the nearest image
        for im in images:
            e = [d[q] - im[q] for q in range(3)]
            r2 = e[0] ** 2 + e[1] ** 2 + e[2] ** 2
            own = r2 == 0
            r2s = r2.clamp(min=1e-24)
            r = r2s.sqrt()
            long_ = torch.erfc(alpha * r) / r
            push = (long_ + 2 * alpha / math.sqrt(math.pi) * torch.exp(-alpha * alpha * r2s)) / r2s
            if im == (0, 0, 0):
                q2 = r2 / (h * h)
                soft = r2 <= h * h
                f = ((((315 / 128 * q2 - 385 / 32) * q2 + 1485 / 64) * q2 - 693 / 32) * q2 + 1155 / 128) / h ** 3
                w = (((((-63 / 256 * q2 + 385 / 256) * q2 - 495 / 128) * q2 + 693 / 128) * q2 - 1155 / 256) * q2 + SELF_PHI) / h
                long_ = torch.where(soft, long_ - 1 / r + w, long_)
                push = torch.where(soft, push - 1 / (r2s * r) + f, push)
                # the particle itself: what the long-range part of its own charge leaves
                long_ = torch.where(own, torch.full_like(r, -2 * alpha / math.sqrt(math.pi)), long_)
                push = torch.where(own, torch.zeros_like(r), push)
            out[3, a:a + step] -= long_.sum(1)
            for q in range(3):
                out[q, a:a + step] -= (e[q] * push).sum(1)
    out[3] += n * math.pi / alpha ** 2
    hs = [(i, j, k) for i in range(-9, 10) for j in range(-9, 10) for k in range(-9, 10) if (i, j, k) > (0, 0, 0) and i * i + j * j + k * k <= 81]
    for a in range(0, len(hs), 256):
        H = torch.tensor(hs[a:a + 256], dtype=torch.float64, device=dev)
        h2 = (H ** 2).sum(1)
        c0 = -2.0 * torch.exp(-math.pi ** 2 * h2 / alpha ** 2) / (math.pi * h2)
        ph = 2 * math.pi * (H @ p)
        C, S = torch.cos(ph), torch.sin(ph)
        cs, sn = C.sum(1, keepdim=True), S.sum(1, keepdim=True)
        out[3] += (c0[:, None] * (C * cs + S * sn)).sum(0)
        out[:3] += (H * (2 * math.pi * c0)[:, None]).t() @ (S * cs - C * sn)
    return out * GM


def _exact_step(case, seed):
    s = prepare(case, seed)  # the inputs
    torch.cuda.synchronize()
    bits = s.x.to(torch.int64) & 0xFFFFFFFF
    order = torch.from_numpy(_tree_order(bits.cpu().numpy(), case["theta"], s.h, case["bucket"])).cuda()
    x, v = s.x[:, order], s.v[order].double()
    g = _exact_gravity(x, s.h, s.GM)
    h, t0 = float(np.float32(s.h)), s.t0
    dt = torch.clamp(ics.eta_default() * (h / g[:3].square().sum(0).sqrt().clamp(min=1e-30)).sqrt(), max=t0)
    up = torch.ceil(torch.log2(t0 / dt)) > 0
    rung = torch.maximum(up.to(torch.int64), s.r[order].to(torch.int64) - 1).clamp(0, 15)
    mid = v + 0.5 * t0 * g[:3].t()
    end = mid + 0.5 * t0 * g[:3].t()
    p = x.double() / 4294967296.0
    p = torch.where((rung == 0)[None], p + end.t() * t0, p)
    p = p - (p >= 0.5).double() + (p < -0.5).double()
    kin = 0.5 * mid.square().sum()
    energy = [kin, 0.5 * (end.square().sum() - v.square().sum())] + [0.5 * g[3].sum()] * case["do_phi"]
    out = {"pos": p, "vel": end, "rung": None, "energy": torch.stack(energy)[None].cpu().numpy(), "max_rung": None,
           "momentum": torch.stack([mid[:, 0].sum(), mid[:, 1].sum(), mid[:, 2].sum(), mid.square().sum(1).sqrt().sum()])[None].cpu().numpy()}
    if case["save_force"]:
        out["force"] = g[:3]
        if case["do_phi"]:
            out["pot"] = g[3]
    return out


def _filter(k):
    """The inverse window of the quintic cloud kernel at wavenumber k (grid units)."""
    return torch.where(k == 0, torch.ones_like(k), torch.sin(0.5 * k) / torch.where(k == 0, torch.ones_like(k), 0.5 * k)) ** -6


def _cloud(t):
    a = t.abs()
    a2, a3 = a ** 2, a ** 3
    inner = (33 - 30 * a2 + 15 * a2 ** 2 - 5 * a2 * a3) / 60
    mid = (51 + 75 * a - 210 * a2 + 150 * a3 - 45 * a2 ** 2 + 5 * a2 * a3) / 120
    outer = (243 - 405 * a + 270 * a2 - 90 * a3 + 15 * a2 ** 2 - a2 * a3) / 120
    return torch.where(a < 1, inner, torch.where(a < 2, mid, torch.where(a <= 3, outer, torch.zeros_like(a))))


def _taus(seed, draws, dev):
    """The first `draws` outputs, as fractions of 2^32, of L'Ecuyer's (1996) Tausworthe generator
    for every seed (n,), seeded as GSL seeds it."""
    M = 0xFFFFFFFF
    s = torch.where(seed == 0, torch.ones_like(seed), seed)
    s1 = (69069 * s) & M
    s2 = (69069 * s1) & M
    s3 = (69069 * s2) & M
    out = torch.empty((draws, seed.numel()), dtype=torch.float64, device=dev)
    for i in range(draws + 6):
        s1 = (((s1 & 4294967294) << 12) & M) ^ ((((s1 << 13) & M) ^ s1) >> 19)
        s2 = (((s2 & 4294967288) << 4) & M) ^ ((((s2 << 2) & M) ^ s2) >> 25)
        s3 = (((s3 & 4294967280) << 17) & M) ^ ((((s3 << 3) & M) ^ s3) >> 11)
        if i >= 6:
            out[i - 6] = (s1 ^ s2 ^ s3).double() / 4294967296.0
    return out


def _log_power(logk, tab):
    logP, k0, dk = tab
    q = (logk - k0) / dk
    i = (q.to(torch.int64) - 1).clamp(0, len(logP) - 4)
    y0, y1, y2, y3 = (logP[i + j] for j in range(4))
    t = q - (i + 1)
    k1, k2 = (y2 - y0) * 0.5, (y3 - y1) * 0.5
    return y1 + k1 * t + (-2 * k1 - k2 - 3 * y1 + 3 * y2) * t ** 2 + (k1 + k2 + 2 * y1 - 2 * y2) * t ** 3


def _growth(om, a):
    a3 = a ** 3
    den = 1.0 / (om + a3 * (1 - om))
    Om, Ol = om * den, a3 * (1 - om) * den
    return a * 2.5 * Om / (Om ** (4 / 7) - Ol + (1 + 0.5 * Om) * (1 + Ol / 70))


def _exact_initialize(case, seed, dev="cuda"):
    N, box, hub = case["grid"], IC_BOX, COSMO["hubble"]
    tk, tp = (torch.from_numpy(np.asarray(t)).to(dev).double() for t in _table(case, seed))
    logk = (tk * hub).log()
    k0, k9 = float(logk.min()), float(logk.max())
    dk = (k9 - k0) / (len(tk) - 1)
    logP = (tp / hub ** 3).log()
    # the table's variance in 8 / h Mpc spheres by Simpson's rule, scaled to sigma8
    M = 8192
    lk = torch.linspace(k0 + 1.5 * dk, k9 - 2.5 * dk, M + 1, dtype=torch.float64, device=dev)
    kk, R = lk.exp(), 8 / hub
    f = 9 / (2 * math.pi ** 2) / R ** 6 * _log_power(lk, (logP, k0, dk)).exp() * ((kk * R).sin() - kk * R * (kk * R).cos()) ** 2 / kk ** 3
    w = torch.full((M + 1,), 2.0 / 3.0, dtype=torch.float64, device=dev)
    w[1::2] = 4.0 / 3.0
    w[0] = w[-1] = 1.0 / 3.0
    logP = logP + math.log(COSMO["sigma8"] ** 2 / float((w * f).sum() * (lk[1] - lk[0])))
    om, a0 = COSMO["omega_m"], 1.0 / (COSMO["z0"] + 1)
    D1 = _growth(om, a0) / _growth(om, 1.0)
    Om = om / (om + a0 ** 3 * (1 - om))
    H = COSMO["H0"] * math.sqrt(om / a0 ** 3 + 1 - om)
    pre = Om ** (5 / 9) * H * a0 * a0, 2 * Om ** (6 / 11) * H * a0 * a0
    D2 = -3 * D1 * D1 / 7
    # the modes' amplitudes: a generator for every (x, y) row, the kz = 0 mode from the mirrored row's
    NZ = N // 2 + 1
    I = torch.arange(N, device=dev)
    J = torch.where(I > N // 2, N - I, I)
    row = (I[:, None] * N + I[None, :]).reshape(-1)
    mir = (J[:, None] * N + J[None, :]).reshape(-1)
    u = _taus((row * 1234 + 42) & 0xFFFFFFFF, 8 + 2 * (NZ - 1), dev)[8:]
    u0 = _taus((mir * 1234 + 42) & 0xFFFFFFFF, 10, dev)[8:]
    U = torch.cat([u0[None], u.view(NZ - 1, 2, -1)]).permute(1, 2, 0).reshape(2, N, N, NZ)
    i1 = torch.where(I < N // 2, I, I - N).double() * (2 * math.pi / box)
    iz = i1[:NZ]
    K = [i1[:, None, None], i1[None, :, None], iz[None, None, :]]
    k2 = K[0] ** 2 + K[1] ** 2 + K[2] ** 2
    k2[0, 0, 0] = 1.0
    size = (-U[0].log()).sqrt() * (0.5 * _log_power(0.5 * k2.log(), (logP, k0, dk))).exp() * box ** -1.5 * N ** 3
    A = torch.polar(size, 2 * math.pi * U[1])
    A[0, 0, 0] = 0
    del u, u0, U, size
    fil = _filter(K[0] * box / N) * _filter(K[1] * box / N) * _filter(K[2] * box / N) / k2
    lower = ((I[:, None] > N // 2) | ((I[:, None] == 0) & (I[None, :] > N // 2)))

    def field(*dims):
        Y = A.clone()
        for d in dims:
            Y = Y * (-1j * K[d])
        Y = Y * fil
        Y[:, :, 0] = torch.where(lower, (-1.0) ** len(dims) * Y[:, :, 0].conj(), Y[:, :, 0])
        return torch.fft.irfftn(Y, s=(N, N, N))

    def smooth(r):
        for d in range(3):  # the kernel at the lattice points
            r = 0.55 * r + 26 / 120 * (r.roll(1, d) + r.roll(-1, d)) + 1 / 120 * (r.roll(2, d) + r.roll(-2, d))
        return r

    pos = torch.stack(torch.meshgrid(I, I, I, indexing="ij")).double().reshape(3, -1) / N
    vel = torch.zeros_like(pos)
    big = []
    for d in range(3):
        dx = smooth(field(d)).reshape(-1) * (-D1 / box)
        pos[d] += dx
        vel[d] += pre[0] * dx
        big.append(float(dx.max()) * N)
    if case["twolpt"]:
        yy, zz, xx = field(1, 1), field(2, 2), field(0, 0)
        src = yy * zz + xx * zz + xx * yy - field(0, 2) ** 2 - field(1, 2) ** 2
        del yy, zz, xx
        k = torch.fft.rfftn(src)
        k[0, 0, 0] = 0
        for d in range(3):
            dx = smooth(torch.fft.irfftn(-1j * K[d] * k * fil, s=(N, N, N))).reshape(-1) * (D2 / box)
            pos[d] += dx
            vel[d] += pre[1] * dx
            big.append(float(dx.max()) * N)
    pos = pos - (pos + 0.5).floor()
    return {"pos": pos, "vel": vel.t(), "rung": None, "dxmax": np.array(big)}


def _exact_power(case, seed):
    x, _ = _particles(case["n"], "clustered", _gen(seed))
    return _power64(x, case["grid"], case["fold"])


def _power64(x, N, fold):
    dev = x.device
    p = (x.to(torch.int64) & 0xFFFFFFFF).double() / 4294967296.0
    p = (p * fold).frac() * N
    cell = p.floor()
    off = p - cell
    cell = cell.to(torch.int64)
    rho = torch.full((N ** 3,), -1.0, dtype=torch.float64, device=dev)
    w = [[_cloud(off[d] - j) for j in range(-2, 4)] for d in range(3)]
    c = [[(cell[d] + j) % N for j in range(-2, 4)] for d in range(3)]
    for a in range(6):
        for b in range(6):
            wab, at = w[0][a] * w[1][b], (c[0][a] * N + c[1][b]) * N
            for q in range(6):
                rho.index_add_(0, at + c[2][q], wab * w[2][q])
    Y = torch.fft.rfftn(rho.view(N, N, N))
    I = torch.arange(N, device=dev)
    i = torch.where(I < N // 2, I, I - N).double()
    k1 = 2 * math.pi * i / N
    f = _filter(k1)
    Y = Y * (f[:, None, None] * f[None, :, None] * f[None, None, : N // 2 + 1])
    kk = (i[:, None, None] ** 2 + i[None, :, None] ** 2 + (i[: N // 2 + 1] ** 2)[None, None, :]).sqrt()
    ns = max(N / 8.0, 64.0)
    l0, l1 = math.log(0.999999), math.log(N / 2.0)
    kb = np.array([math.exp(l0 + (l1 - l0) / ns * q) for q in range(int(ns) + 1)], np.float32)
    edges = torch.from_numpy(kb.astype(np.float64)).to(dev)
    nb = len(kb) - 1
    which = torch.bucketize(kk, edges, right=True) - 1
    # (below the first edge counts in the first bin)
    ok = (kk > 0) & (kk < edges[-1])
    b = which.clamp(min=0)[ok]
    pw = (Y.real ** 2 + Y.imag ** 2)[ok]
    cnt = torch.bincount(b, minlength=nb).double()
    P = torch.bincount(b, weights=pw, minlength=nb) / cnt.clamp(min=1)
    f3 = f.sqrt()  # 1 / sinc^3
    pw2 = (pw * ((f3[:, None, None] * f3[None, :, None] * f3[None, None, : N // 2 + 1]) ** 2).expand_as(kk)[ok])
    dev2 = torch.bincount(b, weights=(pw2 - P[b]) ** 2, minlength=nb)
    err = torch.where(cnt > 1, dev2.sqrt() / (cnt - 1).clamp(min=1).sqrt() / cnt.clamp(min=1).sqrt(), torch.zeros_like(cnt))
    P = torch.where(cnt == 1, torch.zeros_like(P), P)
    kmid = np.sqrt(kb[:-1].astype(np.float64) * kb[1:]) * (2 * math.pi / IC_BOX) * fold
    return {"k": kmid, "P": P.cpu().numpy(), "err": err.cpu().numpy()}
