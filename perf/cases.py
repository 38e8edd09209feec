"""Timed workloads of the framework: runs, host exchanges and training passes.

Every case goes through the public Python binding of the C ABI (rhybrid_b200.abi
and .config). Kinds:

  box      a periodic box stepped on the device, its moments and field read back
  planet   a Mars- or Mercury-like obstacle run filled on the GPU, with its
           particle sources, optionally with the learned denoiser in the step
  output   a closed box with an obstacle, nodeE smoothing, temporal averages,
           constraint counters and log sums, read out at the end of the pass
  exchange a host that owns the particle lists: upload, one step, download
  gradient loss and parameter gradients of the denoiser for host moments
  train    denoiser training on crops stored from a run

`exact` restates the box and exchange kinds and the denoiser's gradient in plain
torch at 64 bits. Runs with particle sources have no such value: the sources
draw from the framework's own random stream.
"""
import math

import numpy as np
import torch

from rhybrid_b200 import abi
from rhybrid_b200 import config as cf

PATHS = {"fast": abi.PATH_FAST, "exact": abi.PATH_EXACT, "fp32": abi.PATH_FP32}
QE, MP, MU0, KB = abi.CHARGE_ELEMENTARY, abi.MASS_PROTON, abi.PERMEABILITY, abi.BOLTZMANN
DN_C, DN_TAPS, DN_LEAK = 16, 27, 0.125
DN_LAYER = DN_TAPS * DN_C * DN_C + DN_C


def listed():
    return [
        # one step of a tiny periodic box and its whole state: launches, synchronisations and copies are all there is
        {"name": "box_tiny", "kind": "box", "path": "fast", "nx": 16, "ny": 16, "nz": 16, "ppc": 8.0, "steps": 1,
         "particles": True},
        # the reference's empty test box (32^3 cells, 20 particles per cell), ten steps between outputs of the whole state
        {"name": "box_32", "kind": "box", "path": "fast", "nx": 32, "ny": 32, "nz": 32, "ppc": 20.0, "steps": 10,
         "particles": True},
        # odd sizes and a fractional particle count per cell on the FP32 form
        {"name": "box_ragged_fp32", "kind": "box", "path": "fp32", "nx": 77, "ny": 53, "nz": 41, "ppc": 12.5, "steps": 4,
         "particles": False},
        # the Mars-like run, FP64, with solar wind and exosphere: the framework's main workload
        {"name": "mars_fp64", "kind": "planet", "planet": "mars", "path": "fast", "nx": 120, "ny": 160, "nz": 160,
         "ppc": 30.0, "steps": 10, "denoise": False},
        # the same run on the FP32 form
        {"name": "mars_fp32", "kind": "planet", "planet": "mars", "path": "fp32", "nx": 120, "ny": 160, "nz": 160,
         "ppc": 30.0, "steps": 10, "denoise": False},
        # the Mercury-like dipole at half its resolution: more cells per ion, so the field update weighs more
        {"name": "mercury_fp64", "kind": "planet", "planet": "mercury", "path": "fast", "nx": 160, "ny": 160, "nz": 160,
         "ppc": 16.0, "steps": 5, "denoise": False},
        # the learned form: 8 particles per cell and the denoiser applied in every step
        {"name": "mars_learned", "kind": "planet", "planet": "mars", "path": "fast", "nx": 120, "ny": 160, "nz": 160,
         "ppc": 8.0, "steps": 5, "denoise": True},
        # a run at its output step: averages, counters and log sums on, E smoothed, odd sizes
        {"name": "output_run", "kind": "output", "nx": 61, "ny": 83, "nz": 70, "ppc": 10.0, "steps": 5, "linear": 1,
         "gauss": 0.8},
        # the reference's particle order, as used to check a set-up against the CPU code
        {"name": "exact_box", "kind": "box", "path": "exact", "nx": 64, "ny": 48, "nz": 40, "ppc": 20.0, "steps": 2,
         "particles": False},
        # a host that owns the particle lists: every ion crosses to the GPU and back around one step
        {"name": "host_exchange", "kind": "exchange", "path": "fast", "nx": 60, "ny": 80, "nz": 80, "ppc": 30.0},
        # the denoiser's backward pass for given moments
        {"name": "dn_gradient", "kind": "gradient", "nx": 64, "ny": 64, "nz": 64, "periodic": False},
        # denoiser training on stored crops of a run
        {"name": "dn_train", "kind": "train", "nx": 64, "ny": 64, "nz": 64, "iterations": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "planet", "planet", "output", "exchange", "gradient", "train"])
    if kind == "box":
        path = rng.choice(["fast", "fast", "fp32", "exact"])
        most = 48 if path == "exact" else 90
        c = {"kind": kind, "path": path, "nx": _log_int(rng, 5, most), "ny": _log_int(rng, 5, most),
             "nz": _log_int(rng, 5, most), "ppc": round(math.exp(rng.uniform(math.log(2.0), math.log(40.0))), 2),
             "steps": rng.randint(1, 8)}
        c["particles"] = path != "fp32" and c["nx"] * c["ny"] * c["nz"] * c["ppc"] < 2e5
        return c
    if kind == "planet":
        planet = rng.choice(["mars", "mercury"])
        path = rng.choice(["fast", "fast", "fp32"])
        lo, hi = (44, 120) if planet == "mars" else (80, 150)
        return {"kind": kind, "planet": planet, "path": path, "nx": rng.randint(lo, hi), "ny": rng.randint(lo, hi),
                "nz": rng.randint(lo, hi), "ppc": round(math.exp(rng.uniform(math.log(4.0), math.log(32.0))), 1),
                "steps": rng.randint(2, 8), "denoise": rng.random() < 0.3}
    if kind == "output":
        return {"kind": kind, "nx": rng.randint(24, 80), "ny": rng.randint(24, 80), "nz": rng.randint(24, 80),
                "ppc": round(rng.uniform(4.0, 20.0), 1), "steps": rng.randint(2, 6), "linear": rng.randint(0, 2),
                "gauss": rng.choice([0.0, 0.8])}
    if kind == "exchange":
        return {"kind": kind, "path": rng.choice(["fast", "exact"]), "nx": rng.randint(12, 60), "ny": rng.randint(12, 60),
                "nz": rng.randint(12, 60), "ppc": round(rng.uniform(3.0, 30.0), 1)}
    if kind == "gradient":
        return {"kind": kind, "nx": rng.randint(9, 64), "ny": rng.randint(9, 64), "nz": rng.randint(9, 64),
                "periodic": rng.random() < 0.5}
    return {"kind": kind, "nx": rng.randint(16, 64), "ny": rng.randint(16, 64), "nz": rng.randint(16, 64),
            "iterations": rng.randint(2, 8)}


# ---------------------------------------------------------------------------
# configurations

def _closed_box(case):
    """Closed walls, an absorbing sphere, H+ and He++, electron pressure, IMF at the +x wall."""
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], 100e3
    R = 0.18 * min(nx, ny, nz) * dx
    pops = [cf.Population(name="H+", obstacle=R, density=2e6, velocity=(-450e3, 0, 0), temperature=1e5, ppc=case["ppc"]),
            cf.Population(name="He++", mass=3.9737, charge=2.0, obstacle=R, density=0.08e6, velocity=(-450e3, 0, 0),
                          temperature=1e5, ppc=max(case["ppc"] / 4, 1.0))]
    return cf.Config(nx=nx, ny=ny, nz=nz, x_min=-0.5 * nx * dx, y_min=-0.5 * ny * dx, z_min=-0.5 * nz * dx, dx=dx,
                     periodic=(0, 0, 0), dt=0.02, R_fieldObstacle=R, R_particleObstacle=R, imf=(0.0, 5e-9, 0.0),
                     imf_boundary_cellB=(1, 0, 0, 0, 0, 0), imf_boundary_faceB=(1, 0, 0, 0, 0, 0),
                     use_electron_pressure=True, electron_temperature=1e5, electron_gamma=2, R_zeroElectronPressure=R,
                     electric_field_linear_smoothing_number=case.get("linear", 0),
                     electric_field_smoothing_gauss_sigma=case.get("gauss", 0.0), populations=pops, name="closed_box")


def _config(case):
    k = case["kind"]
    if k == "box":
        return cf.config_empty_box(case["nx"], case["ny"], case["nz"], ppc=case["ppc"])
    if k == "planet":
        if case["planet"] == "mars":
            return cf.config_mars(case["nx"], case["ny"], case["nz"], ppc=case["ppc"], exosphere=True)
        return cf.config_mercury(case["nx"], case["ny"], case["nz"], ppc=case["ppc"], dx=32000e3 / case["nx"])
    return _closed_box(case)


def _particles(ncells, dx, density, velocity, temperature, mass, ppc, rng):
    """(counts, records) of a uniform Maxwellian fill: 7 doubles per particle, grouped by cell."""
    n = int(round(ppc * ncells))
    counts = np.full(ncells, n // ncells, dtype=np.uint32)
    counts[rng.permutation(ncells)[:n % ncells]] += 1
    p = np.empty((n, 7))
    p[:, :3] = dx * (5e-5 + (1.0 - 1e-4) * rng.random((n, 3)))
    p[:, 3:6] = rng.standard_normal((n, 3)) * math.sqrt(KB * temperature / (mass * MP))
    p[:, 3:6] += np.asarray(velocity, dtype=float)
    p[:, 6] = density * dx ** 3 / ppc
    return counts, p


def _host_particles(cfg, seed):
    rng = np.random.default_rng(seed)
    return [_particles(cfg.ncells, cfg.dx, q.density, q.velocity, q.temperature, q.mass, q.ppc, rng)
            for q in cfg.populations]


def _pinned(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _ptr(t, ct=abi.C.c_double):
    return abi.C.cast(t.data_ptr(), abi.C.POINTER(ct))


# ---------------------------------------------------------------------------
# the denoiser's inputs

def _dn_params(seed, near_identity):
    """Parameters near the untrained pass-through of a run, or a generic network for the gradient."""
    rng = np.random.default_rng(seed)
    p = np.zeros(3 * DN_LAYER, dtype=np.float32)
    for l, (cin, cout) in enumerate(((4, 16), (16, 16), (16, 4))):
        w = np.zeros((DN_TAPS, DN_C, DN_C), dtype=np.float32)
        w[:, :cin, :cout] = rng.standard_normal((DN_TAPS, cin, cout)) * math.sqrt(2.0 / (DN_TAPS * cin))
        if l == 2 and near_identity:
            w *= 0.02
        p[l * DN_LAYER:l * DN_LAYER + w.size] = w.reshape(-1)
        b = 0.05 * rng.standard_normal(cout)
        if l == 2 and near_identity:
            b *= 0.02
        p[l * DN_LAYER + w.size:l * DN_LAYER + w.size + cout] = b
    return p


RHO0, J0 = 3.2e-13, 1.44e-7   # upstream charge density [C m^-3] and current density [A m^-2]


def _moments(case, seed):
    """Noisy moments and their smooth targets: (rho, ji, rho_target, ji_target)."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    z, y, x = np.meshgrid(np.arange(nz) / nz, np.arange(ny) / ny, np.arange(nx) / nx, indexing="ij")
    wave = (1.0 + 0.4 * np.sin(2 * np.pi * (x + 0.7 * y)) * np.cos(2 * np.pi * z)).reshape(-1)
    rho_t = RHO0 * wave
    ji_t = J0 * np.stack([-wave, 0.2 * wave - 0.1, 0.1 * np.cos(2 * np.pi * x).reshape(-1)], axis=1)
    rho = rho_t * (1.0 + 0.2 * rng.standard_normal(n))
    ji = ji_t + 0.2 * J0 * rng.standard_normal((n, 3))
    return rho, ji, rho_t, ji_t


# ---------------------------------------------------------------------------
# prepare and run

def _load_grid(ctx, grid):
    ctx.upload_array("faceB", grid["faceB"])
    ctx.upload_array("cellB", grid["cellB"])
    ctx.upload_array("nodeEta", grid["nodeEta"])
    ctx.upload_cell_flags(grid["flags"])


def prepare(case, seed):
    kind = case["kind"]
    lib = abi.gpu_library()
    st = {"case": case, "lib": lib}
    if kind == "gradient":
        per = (1, 1, 1) if case["periodic"] else (0, 0, 0)
        dn = abi.Denoiser(lib, case["nx"], case["ny"], case["nz"], per)
        dn.set_scales(RHO0, J0)
        dn.set_params(_dn_params(seed, False))
        st.update(dn=dn, moments=_moments(case, seed))
        return st
    if kind == "train":
        # a source run of 1.5 times the crop's size, stepped once, and eight crops of it (1 in 4 of its ions)
        big = [max(int(1.5 * case[a]), case[a] + 4) for a in ("nx", "ny", "nz")]
        cfg = cf.config_empty_box(*big, ppc=16.0)
        dn = abi.Denoiser(lib, case["nx"], case["ny"], case["nz"], (0, 0, 0), pair_capacity=8)
        dn.set_scales(5e6 * QE, 5e6 * QE * 400e3)
        with abi.Context(lib, cf.params(cfg), cf.species(cfg)) as ctx:
            ctx.set_path(abi.PATH_FAST)
            _load_grid(ctx, cf.init_grid(cfg))
            p = cfg.populations[0]
            ctx.fill_uniform(0, p.density, p.temperature, p.velocity, p.ppc, seed=seed + 1)
            ctx.step(1)
            rng = np.random.default_rng(seed)
            o = np.stack([rng.integers(0, b - case[a] + 1, 8) for a, b in zip(("nx", "ny", "nz"), big)], axis=1)
            dn.add_crops(ctx, 4, 1, o)
        dn.set_loss_border(2)
        st.update(dn=dn, params=_dn_params(seed, True))
        return st
    cfg = _config(case)
    ctx = abi.Context(lib, cf.params(cfg), cf.species(cfg))
    ctx.set_path(PATHS[case.get("path", "fast")])
    _load_grid(ctx, cf.init_grid(cfg))
    st.update(ctx=ctx, rho=_pinned(cfg.ncells), ji=_pinned((cfg.ncells, 3)), faceB=_pinned((cfg.ncells, 3)))
    if kind in ("box", "exchange"):
        pops = _host_particles(cfg, seed)
        for s, (cnt, p) in enumerate(pops):
            ctx.upload_particles(s, cnt, p)
        if kind == "exchange":
            st["in"] = [(cnt, _pinned(p.shape)) for cnt, p in pops]
            for (_, hp), (_, p) in zip(st["in"], pops):
                hp.numpy()[:] = p
        st["out"] = [(_pinned(cfg.ncells, torch.int32), _pinned(p.shape)) for _, p in pops]
        return st
    # a run's ion count rises from its fill (pile-up at the obstacle, exospheric ions): storage for that is
    # reserved before the run starts, by a larger fill of every species
    grow = 2.5 if cfg.ncells < 1_000_000 else 1.6
    for s, p in enumerate(cfg.populations):
        if p.ppc > 0 and p.density > 0:
            for f in (grow, 1.0):
                ctx.fill_uniform(s, p.density, p.temperature, p.velocity, f * p.ppc, seed=seed * 101 + s + 1)
        else:
            ctx.fill_uniform(s, 1.0, 1.0, (0.0, 0.0, 0.0), 1.0 + 8e6 / cfg.ncells, seed=1)
            ctx.upload_particles(s, np.zeros(cfg.ncells, dtype=np.uint32), np.zeros((0, 7)))
    ctx.set_injectors(cf.source_injectors(cfg, seed=seed + 1))
    if kind == "output":
        ctx.set_population_averages([0, 1])
        ctx.set_grid_counters(True)
    if case.get("denoise"):
        dn = abi.Denoiser(lib, cfg.nx, cfg.ny, cfg.nz, cfg.periodic)
        p0 = cfg.populations[0]
        rho0 = sum(p.density * p.charge for p in cfg.populations) * QE
        dn.set_scales(rho0, rho0 * abs(p0.velocity[0]))
        dn.set_params(_dn_params(seed, True))
        ctx.set_denoiser(dn)
        st["dn"] = dn
    return st


def _read(st):
    ctx, lib = st["ctx"], st["lib"]
    for name, key in (("cellRhoQi", "rho"), ("cellJi", "ji"), ("faceB", "faceB")):
        lib.call("download_array", ctx.h, abi.ARRAY_ID[name], _ptr(st[key]))
    return {"rho": st["rho"], "ji": st["ji"], "faceB": st["faceB"]}


def _read_ions(st):
    """Every species' counts and records into its host buffers; ions lost since the start leave rows unused."""
    ctx, out = st["ctx"], []
    for s, (cnt, p) in enumerate(st["out"]):
        n = abi.C.c_int64()
        st["lib"].call("download_particles", ctx.h, s, _ptr(cnt, abi.C.c_uint32), _ptr(p), p.shape[0], abi.C.byref(n))
        out.append({"n": n.value, "counts": cnt, "particles": p})
    return out


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "gradient":
        loss, grad = st["dn"].loss_grad(*st["moments"])
        return {"loss": loss, "grad": grad}
    if kind == "train":
        dn = st["dn"]
        dn.set_params(st["params"])
        loss = dn.train(case["iterations"], 1e-3)
        return {"loss": loss, "params": dn.params()}
    ctx = st["ctx"]
    if kind == "exchange":
        for s, (cnt, p) in enumerate(st["in"]):
            ctx.upload_particles(s, cnt, p.numpy())
        ctx.step(1)
        out = _read(st)
        out["species"] = _read_ions(st)
        return out
    ctx.step(case["steps"])
    out = _read(st)
    if kind == "box":
        if case["particles"]:
            out["species"] = _read_ions(st)
        return out
    out["ions"] = [ctx.num_particles(s) for s in range(ctx.nspecies)]
    if kind == "output":
        out["averages"] = ctx.output_averages()
        out["limits"] = ctx.grid_counters()
        d = ctx.reduce_diagnostics(scales=True)
        out["log"] = np.array([v for q in d["populations"] + [d["field"]] for v in q.values()])
    return out


# ---------------------------------------------------------------------------
# work

def _ions(case):
    n = case["nx"] * case["ny"] * case["nz"]
    ppc = case.get("ppc", 0.0)
    if case["kind"] == "planet" and case["planet"] == "mars":
        return n * ppc * 1.05
    if case["kind"] in ("output", "exchange"):
        return n * (ppc + max(ppc / 4, 1.0))
    return n * ppc


def _dn_flops(n):
    return 2.0 * DN_TAPS * (4 * 16 + 16 * 16 + 16 * 4) * n


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind == "gradient":   # moments and targets in, three passes of the network's products
        return {"bytes": 64.0 * n, "flops": 3 * _dn_flops(n)}
    if kind == "train":      # stored crops in, weights out
        return {"bytes": 32.0 * n * case["iterations"], "flops": 3 * _dn_flops(n) * case["iterations"]}
    ions = _ions(case)
    rec = 56 if case.get("path") == "fp32" else 104    # one read and one write of a stored particle
    # per cell and step: faceB, rho, Ji in, faceB, Ue, rho, Ji out, Ep out where there is electron pressure
    cell = 136 + (0 if kind == "box" else 48)
    steps = case.get("steps", 1)
    b = steps * (rec * ions + cell * n) + 56.0 * n
    f = steps * (230.0 * ions + 300.0 * n + (_dn_flops(n) if case.get("denoise") else 0.0))
    if kind == "exchange":
        b += 112.0 * ions
    if case.get("particles"):
        b += 56.0 * ions
    if kind == "output":
        b += 8.0 * n * (3 + 8 + 5)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits

class _Plain:
    """One hybrid step on torch tensors of shape (nz, ny, nx): ions pushed,
    moved and deposited, then the field update (edge currents, upwinded node B,
    Hall term, electron pressure, limiters, Faraday)."""

    def __init__(self, s, dev):
        self.s, self.dev = s, dev
        sh = (s["nz"], s["ny"], s["nx"])
        self.sh = sh
        t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev).reshape(sh)  # noqa: E731
        self.faceB = [torch.full(sh, b, dtype=torch.float64, device=dev) for b in s["imf"]]
        self.cellB = [b.clone() for b in self.faceB]
        self.eta, self.fl = t(s["eta"]), {k: t(v) > 0 for k, v in s["flags"].items()}
        z = torch.zeros(sh, dtype=torch.float64, device=dev)
        self.ue, self.ep = [z.clone() for _ in range(3)], [z.clone() for _ in range(3)]
        self.node_rho = z.clone()
        per = s["periodic"]
        k, j, i = torch.meshgrid(*[torch.arange(n, device=dev) for n in sh], indexing="ij")
        nn = (s["nx"], s["ny"], s["nz"])
        lo = [torch.ones(sh, dtype=torch.bool, device=dev) if per else c > 0 for c in (i, j, k)]
        hi = [torch.ones(sh, dtype=torch.bool, device=dev) if per else c < n - 1 for c, n in zip((i, j, k), nn)]
        self.lo, self.hi = lo, hi
        self.plus = hi[0] & hi[1] & hi[2]
        self.inner = self.plus & lo[0] & lo[1] & lo[2]
        self.wall_x = ~hi[0]
        # nearest inner cell, with some axes left as they are (a face's own axis)
        self.clamped = {}
        for keep in (None, 0, 1, 2):
            c = [x if (per or a == keep) else x.clamp(1, n - 2) for a, (x, n) in enumerate(zip((i, j, k), nn))]
            self.clamped[keep] = (c[2] * nn[1] + c[1]) * nn[0] + c[0]

    def at(self, a, dx=0, dy=0, dz=0):
        return torch.roll(a, (-dz, -dy, -dx), (0, 1, 2))

    def near(self, a, keep=None):
        return a.reshape(-1)[self.clamped[keep]]

    def corner_mean(self, a, sgn):
        at = lambda x, y, z: self.at(a, sgn * x, sgn * y, sgn * z)  # noqa: E731
        return 0.125 * (at(0, 0, 0) + at(0, 0, 1) + at(0, 1, 0) + at(1, 0, 0) + at(0, 1, 1) + at(1, 1, 0) + at(1, 0, 1)
                        + at(1, 1, 1))

    def ions(self, pops):
        s = self.s
        dx, dt, nn, per = s["dx"], s["dt"], (s["nx"], s["ny"], s["nz"]), s["periodic"]
        N = nn[0] * nn[1] * nn[2]
        tot = [torch.zeros(N, dtype=torch.float64, device=self.dev) for _ in range(4)]
        flat = lambda a: a.reshape(-1)  # noqa: E731
        for pop in pops:
            c, x, v, w = pop["c"], pop["x"], pop["v"], pop["w"]
            lin = (c[2] * nn[1] + c[1]) * nn[0] + c[0]
            B = []
            for a in range(3):
                d = [0, 0, 0]
                d[a] = -1
                f = x[a] / dx
                B.append(f * flat(self.faceB[a])[lin] + (1.0 - f) * flat(self.at(self.faceB[a], *d))[lin])
            U = [flat(u)[lin] for u in self.ue]
            E = [B[1] * U[2] - B[2] * U[1], B[2] * U[0] - B[0] * U[2], B[0] * U[1] - B[1] * U[0]]
            E = [e + flat(p)[lin] for e, p in zip(E, self.ep)]
            qm = 0.5 * pop["q"] * dt / pop["m"]
            t = [qm * b for b in B]
            b2 = 2.0 / (1.0 + t[0] ** 2 + t[1] ** 2 + t[2] ** 2)
            vm = [a + qm * e for a, e in zip(v, E)]
            cross = lambda a, b: [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]  # noqa: E731
            v0 = [a + b for a, b in zip(vm, cross(vm, t))]
            vp = [a + b2 * b for a, b in zip(vm, cross(v0, t))]
            vn = [a + qm * e for a, e in zip(vp, E)]
            v2 = vn[0] ** 2 + vn[1] ** 2 + vn[2] ** 2
            fac = torch.where(v2 > s["max_vi2"], torch.sqrt(s["max_vi2"] / v2), torch.ones_like(v2))
            acc = flat(self.inner)[lin]
            v = [torch.where(acc, a * fac, b) for a, b in zip(vn, v)]
            x, cc, ok = [a + dt * b for a, b in zip(x, v)], [], torch.ones_like(acc)
            for a in range(3):
                down, up = x[a] < 0, x[a] >= dx
                x[a] = torch.where(down, x[a] + dx, torch.where(up, x[a] - dx, x[a]))
                x[a] = torch.where(down & (x[a] >= dx), torch.full_like(x[a], np.nextafter(dx, 0.0)), x[a])
                ok &= (x[a] >= 0) & (x[a] < dx)
                ca = c[a] - down.to(c[a].dtype) + up.to(c[a].dtype)
                if per:
                    ca = ca % nn[a]
                else:
                    ok &= (ca >= 0) & (ca < nn[a])
                cc.append(ca)
            c, x, v, w = [a[ok] for a in cc], [a[ok] for a in x], [a[ok] for a in v], w[ok]
            base = [a - (b < 0.5 * dx).to(a.dtype) for a, b in zip(c, x)]
            frac = [torch.where(b < 0.5 * dx, b + 0.5 * dx, b - 0.5 * dx) / dx for b in x]
            for o in range(8):
                wt, idx, inside = w * pop["q"], [], torch.ones_like(w, dtype=torch.bool)
                for a in range(3):
                    up = (o >> a) & 1
                    wt = wt * (frac[a] if up else 1.0 - frac[a])
                    ia = base[a] + up
                    if per:
                        ia = ia % nn[a]
                    else:
                        inside &= (ia >= 0) & (ia < nn[a])
                    idx.append(ia)
                wt = torch.where(inside, wt, torch.zeros_like(wt))
                lin = ((idx[2] * nn[1] + idx[1]) * nn[0] + idx[0]).clamp(0, N - 1)
                lin = torch.where(inside, lin, torch.zeros_like(lin))
                tot[0].index_add_(0, lin, wt)
                for l in range(3):
                    tot[1 + l].index_add_(0, lin, wt * v[l])
            lin = (c[2] * nn[1] + c[1]) * nn[0] + c[0]
            keep = flat(self.inner)[lin]
            if s["R2"] > 0:
                r2 = sum((o + a.to(torch.float64) * dx + b) ** 2 for o, a, b in zip(s["origin"], c, x))
                keep &= ~(flat(self.fl["particle"])[lin] & (r2 < s["R2"]))
            pop.update(c=[a[keep] for a in c], x=[a[keep] for a in x], v=[a[keep] for a in v], w=w[keep])
        dV = dx ** 3
        self.rho = (tot[0] / dV).reshape(self.sh).clamp(min=s["min_rho"])
        self.ji = [(a / dV).reshape(self.sh) for a in tot[1:]]

    def fields(self):
        s, at = self.s, self.at
        dx = s["dx"]
        d = [(-1, 0, 0), (0, -1, 0), (0, 0, -1)]
        self.cellB = [torch.where(self.inner, 0.5 * (f + at(f, *d[a])), b)
                      for a, (f, b) in enumerate(zip(self.faceB, self.cellB))]
        if not s["periodic"]:
            self.cellB, self.ji = [self.near(b) for b in self.cellB], [self.near(j) for j in self.ji]
            self.rho = self.near(self.rho)
            self.faceB = [self.near(f, a) for a, f in enumerate(self.faceB)]
            imf = [torch.full_like(self.rho, b) for b in s["imf"]]
            self.cellB = [torch.where(self.wall_x, m, b) for m, b in zip(imf, self.cellB)]
            self.faceB = [f if a == 0 else torch.where(self.wall_x, m, f)
                          for a, (m, f) in enumerate(zip(imf, self.faceB))]
        f = self.faceB
        Bm = [self.corner_mean(b, 1) for b in self.cellB]
        rho, ji = self.corner_mean(self.rho, 1), [self.corner_mean(j, 1) for j in self.ji]
        curl = []
        for a in range(3):
            b, c = (a + 1) % 3, (a + 2) % 3
            eb, ec, ea = [[int(q == r) for q in range(3)] for r in (b, c, a)]
            e = at(f[c], *eb) - f[c] - at(f[b], *ec) + f[b]
            curl.append(e + at(e, *ea))
        Bt = torch.sqrt(sum(b * b for b in Bm))
        vw = 2.0 * Bt * math.pi / (MU0 * rho * dx)
        lim = torch.where((rho > 0) & (vw > s["max_vw"]), vw / s["max_vw"], torch.ones_like(vw))
        J = [c * 0.5 / (dx * MU0 * lim) for c in curl]
        rc = rho.clamp(min=s["min_rho"])
        ue = self.limit([-(a - b) / rc for a, b in zip(J, ji)], s["max_ue2"])
        ue = [torch.where(self.fl["node"], torch.zeros_like(u), u) for u in ue]
        U = torch.sqrt(sum(u * u for u in ue))
        h = [torch.where(U > 0, -0.5 * u / U.clamp(min=1e-300), z) for u, z in
             zip(ue, (torch.full_like(U, -0.5), torch.zeros_like(U), torch.zeros_like(U)))]
        sw, B = torch.zeros_like(U), [torch.zeros_like(U) for _ in range(3)]
        for o in range(8):
            e = [(o >> a) & 1 for a in range(3)]
            w = 1.0 / torch.sqrt(sum((q - 0.5 - g) ** 2 for q, g in zip(e, h)))
            sw = sw + w
            B = [b + w * at(q, *e) for b, q in zip(B, self.cellB)]
        B = [b / sw for b in B]
        E = [-(ue[1] * B[2] - ue[2] * B[1]), -(ue[2] * B[0] - ue[0] * B[2]), -(ue[0] * B[1] - ue[1] * B[0])]
        E = [torch.where(self.plus, e + self.eta * j, torch.zeros_like(e)) for e, j in zip(E, J)]
        J = [torch.where(self.plus, j, torch.zeros_like(j)) for j in J]
        rn = torch.where(self.plus, rc, self.node_rho)
        self.node_rho = rn
        Jc = [self.corner_mean(j, -1) for j in J]
        u = self.limit([-(a - b) / self.rho for a, b in zip(Jc, self.ji)], s["max_ue2"])
        u = [torch.where(self.fl["field"], torch.zeros_like(a), a) for a in u]
        self.ue = [torch.where(self.inner, a, b) for a, b in zip(u, self.ue)]
        if s["ep"] > 0:
            for a in range(3):
                b, c = [r for r in range(3) if r != a]
                eb, ec, ea = [[-int(q == r) for q in range(3)] for r in (b, c, a)]
                face = 0.25 * (rn + at(rn, *eb) + at(rn, *ec) + at(rn, *[p + q for p, q in zip(eb, ec)]))
                g = -s["ep"] * (face - at(face, *ea)) / dx
                g = torch.where(self.fl["ep"], torch.zeros_like(g), g)
                self.ep[a] = torch.where(self.inner, g, self.ep[a])
        new = []
        for a in range(3):   # dB/dt = -curl E on the face normal to a, from its four nodes
            b, c = (a + 1) % 3, (a + 2) % 3
            eb, ec = [[-int(q == r) for q in range(3)] for r in (b, c)]
            ez, ey = E[c] + at(E[c], *ec), E[b] + at(E[b], *eb)
            curlE = 0.5 * ((ez - at(ez, *eb)) - (ey - at(ey, *ec))) / dx
            on = self.plus & self.lo[b] & self.lo[c]
            new.append(torch.where(on, f[a] - s["dt"] * curlE, f[a]))
        self.faceB = new
        if not s["periodic"]:
            self.ue = [self.near(a) for a in self.ue]

    @staticmethod
    def limit(u, m2):
        u2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        fac = torch.where(u2 > m2, torch.sqrt(m2 / u2), torch.ones_like(u2))
        return [a * fac for a in u]


def _plain_setup(case):
    """The numbers of a box or exchange case, from its definition."""
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], 100e3
    periodic = case["kind"] == "box"
    dt, U = (0.01, 400e3) if periodic else (0.02, 450e3)
    pops = ([{"n": 5e6, "m": MP, "q": QE, "ppc": case["ppc"]}] if periodic else
            [{"n": 2e6, "m": MP, "q": QE, "ppc": case["ppc"]},
             {"n": 0.08e6, "m": 3.9737 * MP, "q": 2.0 * QE, "ppc": max(case["ppc"] / 4, 1.0)}])
    rhoq = sum(p["n"] * p["q"] for p in pops)
    R = 0.0 if periodic else 0.18 * min(nx, ny, nz) * dx
    origin = (-0.5 * nx * dx, -0.5 * ny * dx, -0.5 * nz * dx)
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    rc2 = sum((o + a * dx + 0.5 * dx) ** 2 for o, a in zip(origin, (i, j, k)))
    rn2 = sum((o + a * dx + dx) ** 2 for o, a in zip(origin, (i, j, k)))
    shell = (np.sqrt(rc2) - 0.5 * math.sqrt(3) * dx) ** 2 < R * R
    flags = {"field": rc2 < R * R, "node": rn2 < R * R, "particle": shell, "ep": shell}
    vmax = min(1500e3, 0.9 * dx / dt) if 1500e3 > dx / dt else 1500e3
    return {"nx": nx, "ny": ny, "nz": nz, "dx": dx, "dt": dt, "periodic": periodic, "imf": (0.0, 5e-9, 0.0),
            "origin": origin, "R2": R * R, "flags": flags, "eta": np.full(rc2.shape, MU0 * dx * U / 6.0),
            "max_vi2": vmax ** 2, "max_ue2": 1500e3 ** 2, "max_vw": 1500e3, "min_rho": 0.05 * rhoq,
            "ep": 0.0 if periodic else 2.0 * KB * 1e5 / (rhoq / QE * QE * QE), "pops": pops, "U": (-U, 0.0, 0.0)}


def _exact_run(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    s = _plain_setup(case)
    rng = np.random.default_rng(seed)
    nx, ny = s["nx"], s["ny"]
    pops = []
    for p in s["pops"]:
        cnt, rec = _particles(nx * ny * s["nz"], s["dx"], p["n"], s["U"], 1e5, p["m"] / MP, p["ppc"], rng)
        lin = torch.as_tensor(np.repeat(np.arange(cnt.size), cnt), device=dev)
        r = torch.as_tensor(rec, device=dev).T.contiguous()
        pops.append({"q": p["q"], "m": p["m"], "c": [lin % nx, lin // nx % ny, lin // (nx * ny)],
                     "x": [r[0], r[1], r[2]], "v": [r[3], r[4], r[5]], "w": r[6]})
    sim = _Plain(s, dev)
    for _ in range(case.get("steps", 1)):
        sim.ions(pops)
        sim.fields()
    vec = lambda a: torch.stack([x.reshape(-1) for x in a], dim=1).cpu()  # noqa: E731
    out = {"rho": sim.rho.reshape(-1).cpu(), "ji": vec(sim.ji), "faceB": vec(sim.faceB)}
    if case["kind"] == "exchange" or case["particles"]:
        out["species"] = [{"n": None, "counts": None, "particles": None} for _ in pops]
    return out


def _exact_gradient(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rho, ji, rho_t, ji_t = _moments(case, seed)
    vol = lambda r, j: torch.as_tensor(np.concatenate([r[:, None] / RHO0, j / J0], axis=1), dtype=torch.float64,  # noqa: E731
                                       device=dev).T.reshape(1, 4, nz, ny, nx)
    x, target = vol(rho, ji), vol(rho_t, ji_t)
    p = torch.as_tensor(_dn_params(seed, False).astype(np.float64), device=dev).requires_grad_()
    a = x
    for l in range(3):
        w = p[l * DN_LAYER:l * DN_LAYER + DN_TAPS * DN_C * DN_C].reshape(3, 3, 3, DN_C, DN_C)
        b = p[l * DN_LAYER + DN_TAPS * DN_C * DN_C:(l + 1) * DN_LAYER]
        if a.shape[1] < DN_C:
            a = torch.nn.functional.pad(a, (0, 0, 0, 0, 0, 0, 0, DN_C - a.shape[1]))
        a = torch.nn.functional.pad(a, (1,) * 6, mode="circular" if case["periodic"] else "constant")
        acc = b.reshape(1, DN_C, 1, 1, 1)
        for t in range(DN_TAPS):
            tx, ty, tz = t % 3, t // 3 % 3, t // 9
            acc = acc + torch.einsum("bcdhw,co->bodhw", a[:, :, tz:tz + nz, ty:ty + ny, tx:tx + nx], w[tz, ty, tx])
        a = acc if l == 2 else torch.where(acc > 0, acc, DN_LEAK * acc)
    loss = ((a[:, :4] + x - target) ** 2).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": p.grad.cpu().numpy()}


def exact(case, seed):
    if case["kind"] in ("box", "exchange"):
        return _exact_run(case, seed)
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    return None
