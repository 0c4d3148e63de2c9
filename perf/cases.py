"""The work a user of this framework has it do, as timed cases.

Three kinds of case, each through the public Python entry points:

  steps      one or many boxes advanced by `steps` velocity-Verlet steps (`System.step`, the
             driver loop), then the state read out in original particle order, as a run does
             between two outputs;
  methods    the class_system call sequence, step by step, with the wall forces and the
             kinetic energy read back every step (the drop-in use);
  surrogate  the sweep's network: training steps, or prediction of a set of sweep points.

Boxes start from the lattice the engine builds, disordered as a developed flow is: fluid
particles moved by up to 0.1 lattice spacings, random velocities and a conformation tensor
around the identity, all from the seed.  FP64 states come back as FP64 arrays; states of
mixed-precision runs (float pair terms) as FP32 ones, which is how such a run is kept.

`exact` advances the same inputs in FP64 with plain torch: brute neighbour pairs from its own
cell grid, index_add sums, every box of an ensemble at once.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sph-magnetic-particles-oldroyd-b-in-cuda_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import sph_b200  # noqa: E402
import sph_ensemble  # noqa: E402
import sph_input  # noqa: E402
import sph_surrogate  # noqa: E402

DEV = "cuda:0"
F64 = torch.float64


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest real run: a 2D Kolmogorov box, where launches and latency are all
        dict(name="kolmogorov64", kind="steps", flow="kolmogorov", dim=2, nx=64, ny=64, nz=1,
             overlap=4, boxes=1, colloids=0, precision="fp64", steps=10),
        # a small 2D channel of uneven sides with moving walls, a body force and colloids
        dict(name="channel2d_colloids", kind="steps", flow="channel", dim=2, nx=93, ny=67, nz=1,
             overlap=3, boxes=1, colloids=4, precision="fp64", steps=10),
        # a small, ragged 3D Couette box in mixed precision
        dict(name="couette3d_small_mixed", kind="steps", flow="couette", dim=3, nx=25, ny=19, nz=31,
             overlap=3, boxes=1, colloids=0, precision="mixed", steps=10),
        # an ordinary 3D run: periodic box, opposed body force, odd sides
        dict(name="periodic3d_61", kind="steps", flow="poiseuille", dim=3, nx=61, ny=53, nz=67,
             overlap=3, boxes=1, colloids=0, precision="fp64", steps=5),
        # the drop-in call sequence on an ordinary 3D box
        dict(name="methods3d_48", kind="methods", flow="couette", dim=3, nx=48, ny=48, nz=48,
             overlap=3, boxes=1, colloids=0, precision="fp64", steps=4),
        # the 3D suspension of rotating magnetic colloids
        dict(name="suspension96", kind="steps", flow="suspension", dim=3, nx=96, ny=96, nz=96,
             overlap=3, boxes=1, colloids=32, precision="fp64", steps=5),
        # the largest box of the configurations, in both precisions
        dict(name="couette128", kind="steps", flow="couette", dim=3, nx=128, ny=128, nz=128,
             overlap=3, boxes=1, colloids=0, precision="fp64", steps=5),
        dict(name="couette128_mixed", kind="steps", flow="couette", dim=3, nx=128, ny=128, nz=128,
             overlap=3, boxes=1, colloids=0, precision="mixed", steps=5),
        # a parameter sweep: hundreds of 2D boxes of uneven size in one context
        dict(name="ensemble512", kind="steps", flow="sweep", dim=2, nx=0, ny=0, nz=1, overlap=4,
             boxes=512, colloids=24, precision="fp64", steps=4),
        dict(name="ensemble512_mixed", kind="steps", flow="sweep", dim=2, nx=0, ny=0, nz=1,
             overlap=4, boxes=512, colloids=24, precision="mixed", steps=4),
        # the surrogate: training steps on batches, and the prediction of a sweep's points
        dict(name="surrogate_train", kind="train", heads=5, batch=1024, steps=8),
        dict(name="surrogate_predict", kind="predict", heads=5, points=20011),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: 2D boxes of side 32..192, 3D boxes of side 16..128 (a
    box never larger than the largest listed one), sweeps of 8..512 boxes, batches of the
    surrogate in multiples of 128 up to 1024, and 500..60,000 points to predict."""
    kind = rng.choice(["steps2d", "steps3d", "steps3d", "suspension", "sweep", "methods",
                       "train", "predict"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "steps2d":
        flow = rng.choice(["kolmogorov", "channel", "couette"])
        nx, ny = _log_int(rng, 32, 192), _log_int(rng, 32, 192)
        # the colloids' coarse grid needs three cells of 20 spacings per side
        colloids = 4 if flow == "channel" and min(nx, ny) >= 64 else 0
        return dict(kind="steps", flow=flow, dim=2, nx=nx, ny=ny, nz=1,
                    overlap=rng.choice([3, 4]), boxes=1, colloids=colloids, precision=prec,
                    steps=10)
    if kind == "steps3d":
        flow = rng.choice(["couette", "poiseuille"])
        return dict(kind="steps", flow=flow, dim=3, nx=_log_int(rng, 16, 126),
                    ny=_log_int(rng, 16, 126), nz=_log_int(rng, 16, 126), overlap=3, boxes=1,
                    colloids=0, precision=prec, steps=5)
    if kind == "suspension":
        n = _log_int(rng, 85, 96)  # three coarse colloid cells of 28 spacings per side
        return dict(kind="steps", flow="suspension", dim=3, nx=n, ny=n, nz=n, overlap=3, boxes=1,
                    colloids=rng.randint(2, 32), precision=prec, steps=5)
    if kind == "sweep":
        return dict(kind="steps", flow="sweep", dim=2, nx=0, ny=0, nz=1, overlap=4,
                    boxes=_log_int(rng, 8, 500), colloids=24, precision=prec, steps=4)
    if kind == "methods":
        d = rng.choice([2, 3])
        n = [_log_int(rng, 32, 160) if d == 2 else _log_int(rng, 16, 80) for _ in range(3)]
        return dict(kind="methods", flow="couette", dim=d, nx=n[0], ny=n[1],
                    nz=n[2] if d == 3 else 1, overlap=3, boxes=1, colloids=0, precision=prec,
                    steps=4)
    if kind == "train":
        return dict(kind="train", heads=rng.randint(1, 6), batch=128 * rng.randint(1, 8),
                    steps=rng.randint(4, 10))
    return dict(kind="predict", heads=rng.randint(1, 6), points=_log_int(rng, 500, 60000))


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _specs(case):
    """The `input` keys of every box of a case.  A sweep's points (sides, colloid placements and
    physical parameters) are the same for every seed, which gives the boxes' starts."""
    flow, dim, ov = case["flow"], case["dim"], float(case["overlap"])
    if flow == "sweep":
        pts = sph_ensemble.draw_points(case["boxes"], seed=0)
        return [sph_ensemble.box_spec(p) for p in pts]
    N = (case["nx"], case["ny"], case["nz"])[:dim]
    dx = 1.0 / max(N)
    L = tuple(n * dx for n in N)
    base = dict(N=N, L=L, dim=dim, overlap=ov, dt=2e-5)
    if flow == "kolmogorov":
        return [dict(base, dt=5e-5, ext_force_type=2, ext_force=(1.0, 0.0))]
    if flow == "poiseuille":
        return [dict(base, ext_force_type=3, ext_force=(1.0, 0.0, 0.0)[:dim])]
    if flow == "couette":
        return [dict(base, wall=1, Vwall_bottom=-0.5, Vwall_top=0.5)]
    if flow == "suspension":
        return [sph_input.suspension_spec(N=case["nx"], n_colloids=case["colloids"],
                                          F0_repulsion=1e-3, F0_magnetic=5e-4)]
    assert flow == "channel"
    spec = dict(base, wall=1, Vwall_bottom=-0.2, Vwall_top=0.2, ext_force_type=1,
                ext_force=(0.5, 0.0, 0.0)[:dim])
    if case["colloids"]:
        R = 4.0 * dx
        at = ((0.18, 0.5), (0.36, 0.34), (0.62, 0.62), (0.84, 0.4))[:case["colloids"]]
        spec.update(N_colloids=len(at), coll_R=R, coll_x=tuple((x * L[0], y * L[1]) for x, y in at),
                    coll_repulsion_cuton=0.05 * R, F0_repulsion=1e-3, tau_repulsion=3.0,
                    cutoff_magnetic=5.0 * R, F0_magnetic=1e-4, omega_magnetic=2.0 * math.pi)
    return [spec]


def _disorder(specs, seed, fluid, box, pos):
    """Positions, velocities and conformation tensor of the disordered start, as a dict of
    FP64 arrays over all particles (walls and colloid particles keep their lattice state)."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    n, dim = fluid.shape[0], specs[0]["dim"]
    spacing = torch.tensor([s["L"][0] / s["N"][0] for s in specs], dtype=F64, device=DEV)[box]

    def uniform(scale):
        u = torch.rand(n, generator=g, device=DEV, dtype=F64) * 2.0 - 1.0
        return torch.where(fluid, u * scale, torch.zeros_like(u))

    out = {}
    for k, q in enumerate("xyz"[:dim]):
        out[q] = pos[k] + uniform(0.1 * spacing)
    for q in "xyz"[:dim]:
        out["v" + q] = uniform(0.1)
    diag = ("cxx", "cyy", "czz")[:dim]
    for q in ("cxx", "cxy", "cyy", "cxz", "cyz", "czz")[:3 if dim == 2 else 6]:
        out[q] = uniform(0.1) + (1.0 if q in diag else 0.0)
    return out


class _Boxes:
    """An opened System with its disordered start and the buffers its outputs go to."""

    def __init__(self, case, seed):
        specs = _specs(case)
        self.case, self.dim = case, case["dim"]
        with tempfile.TemporaryDirectory() as wd:
            paths = [sph_input.write_input(os.path.join(wd, "input_%05d" % k), **s)
                     for k, s in enumerate(specs)]
            self.system = s = sph_b200.System(paths, precision=case["precision"])
        sizes = torch.tensor([s.info(b)["N"] for b in range(s.nboxes)], device=DEV)
        box = torch.repeat_interleave(torch.arange(s.nboxes, device=DEV), sizes)
        fluid = torch.from_numpy(s.type()).to(DEV) == 0
        pos = [torch.from_numpy(s.field(q)).to(DEV) for q in "xyz"[:self.dim]]
        start = _disorder(specs, seed, fluid, box, pos)
        keep = torch.stack([torch.where(fluid, start[q], torch.from_numpy(s.field(q)).to(DEV))
                            for q in start if q[0] == "c"]).cpu().numpy()
        for q in start:
            if q[0] != "c":
                s.set_field(q, start[q].cpu().numpy())
        for q, v in zip([q for q in start if q[0] == "c"], keep):
            s.set_field(q, v)
        s.initial_forces()
        self.fields = list(start) + ["fx", "fy", "fz"][:self.dim] + ["dens"]
        if case["kind"] == "methods":
            self.fields += ["press"] + ["g%s%s" % (a, b) for a in "xyz"[:self.dim]
                                        for b in "xyz"[:self.dim]]
        self.buf = torch.empty(len(self.fields), s.N, dtype=F64, device=DEV)

    def read(self):
        """Every field in original order, plus the colloids' state and the wall forces."""
        s, lib = self.system, sph_b200.lib()
        for k, q in enumerate(self.fields):
            s._ok(lib.sph_read_field_device(s._h, sph_b200.FIELDS.index(q),
                                            self.buf[k].data_ptr()))
        out = {}
        if s.ncoll:
            names = [q for q in sph_b200.COLLOID_FIELDS if self.dim == 3 or _in_2d(q)]
            if self.dim == 3:
                names.remove("coll_theta")
            out["colloids"] = np.stack([s.colloid_field(q) for q in names])
        if s.info(0)["wall"]:
            out["walls"] = s.wall_forces()[:, :, :self.dim]
        s.synchronize()
        out["fields"] = {q: self.buf[k] for k, q in enumerate(self.fields)}
        if self.case["precision"] == "mixed":
            out = {k: ({q: t.float() for q, t in v.items()} if isinstance(v, dict)
                       else v.astype(np.float32)) for k, v in out.items()}
        return out


def _in_2d(q):
    return q not in ("coll_z", "coll_vz", "coll_omegax", "coll_omegay", "coll_quat0",
                     "coll_quatx", "coll_quaty", "coll_quatz", "fz_colloid", "tx_colloid",
                     "ty_colloid")


def _network(case, seed):
    """Parameters of every head (He-scaled normal weights, small biases), inputs and targets."""
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    I, H, O = sph_surrogate.IN, sph_surrogate.HID, sph_surrogate.OUT
    parts = []
    for rows, cols in ((H, I), (H, H), (H, H), (O, H)):
        parts.append(torch.randn(case["heads"], rows * cols, generator=g) * math.sqrt(1.5 / cols))
        parts.append(torch.randn(case["heads"], rows, generator=g) * 0.05)
    params = torch.cat(parts, dim=1)
    n = case["points"] if case["kind"] == "predict" else case["steps"] * case["batch"]
    x = torch.randn(n, I, generator=g)
    y = torch.stack([torch.tanh(x[:, 0] + 0.5 * x[:, 1]), x[:, 2] * x[:, 3],
                     torch.sin(x[:, 4]), 0.3 * x[:, 5] + 0.1 * x[:, 0] * x[:, 1]], dim=1)
    return params, x, y


def prepare(case, seed):
    if case["kind"] in ("steps", "methods"):
        return _Boxes(case, seed)
    params, x, y = _network(case, seed)
    net = sph_surrogate.MLP(heads=case["heads"], max_batch=case.get("batch", 1024))
    net.set_params(params.numpy())
    x, y = x.to(DEV), y.to(DEV)
    if case["kind"] == "predict":
        return dict(case=case, net=net, x=x)
    return dict(case=case, net=net, x=x.split(case["batch"]), y=y.split(case["batch"]))


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def run(state):
    if isinstance(state, _Boxes):
        s, n = state.system, state.case["steps"]
        if state.case["kind"] == "steps":
            s.step(n)
            return state.read()
        walls, energy = [], []
        for _ in range(n):
            s.V_Verlet_step1()
            s.neighbours_search()
            s.calculate_forces()
            s.V_Verlet_step2()
            walls.append(s.wall_forces()[:, :, :state.dim])
            energy.append(s.kinetic_energy())
        out = state.read()
        if state.case["precision"] == "fp64":
            out["cells"] = {k: v for k, v in s.export_cells().items() if k.startswith("particle")}
        kind = np.float64 if state.case["precision"] == "fp64" else np.float32
        out["wall_series"] = np.stack(walls).astype(kind)
        out["energy_series"] = np.stack(energy).astype(kind)
        return out
    net = state["net"]
    if state["case"]["kind"] == "predict":
        return net.predict(state["x"])
    for x, y in zip(state["x"], state["y"]):
        net.train_step(x, y, 1e-3)
    return net.get_params()


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _counts(case):
    """(particles, neighbours of a particle inside the cutoff) of a case's boxes."""
    ov, dim = case["overlap"], case["dim"]
    near = math.pi * ov ** 2 if dim == 2 else 4.0 / 3.0 * math.pi * ov ** 3
    if case["flow"] == "sweep":
        # sides of 32..128 spacings, 2 x 4 wall rows each; the drawn points' mean
        return case["boxes"] * 8100, near
    ny = case["ny"]
    if case["flow"] in ("couette", "channel", "suspension"):
        ny += 2 * ov
    return case["nx"] * ny * (case["nz"] if dim == 3 else 1), near


def work(case):
    """Bytes: per step, position, velocity, conformation tensor, force and its rate read and
    written once per particle, and the type word.  Operations: per pair inside the cutoff one
    kernel value and one pair term; the network's multiply-adds for the surrogate."""
    if case["kind"] in ("steps", "methods"):
        n, near = _counts(case)
        d = case["dim"]
        comps = 3 if d == 2 else 6
        per = 2 * 8 * (3 * d + 2 * comps) + 8 + 4
        pair = 30 + (75 if d == 2 else 110)
        return {"bytes": float(n * per * case["steps"]),
                "flops": float(n * near * pair * case["steps"])}
    I, H, O = sph_surrogate.IN, sph_surrogate.HID, sph_surrogate.OUT
    macs = I * H + 2 * H * H + H * O
    params = macs + 3 * H + O
    if case["kind"] == "predict":
        n = case["points"]
        return {"bytes": 4.0 * (n * I + case["heads"] * (n * O + params)),
                "flops": 2.0 * macs * n * case["heads"]}
    n = case["steps"] * case["batch"]
    # weights and both Adam moments read and written once per step
    return {"bytes": 4.0 * (n * (I + O) + 6 * case["heads"] * params * case["steps"]),
            "flops": 6.0 * macs * n * case["heads"]}


# ---------------------------------------------------------------------------------------
# the same in FP64, plain torch
# ---------------------------------------------------------------------------------------
SYM = {(0, 0): 0, (0, 1): 1, (1, 1): 2, (0, 2): 3, (1, 2): 4, (2, 2): 5}


def _sym(c, a, b):
    return c[SYM[(min(a, b), max(a, b))]]


class _Exact:
    """Every box of a case at once; arrays are [component, particle]."""

    CHUNK = 60_000_000  # candidate pairs looked at together

    def __init__(self, case, seed):
        full = [dict(sph_input.DEFAULTS, **s) for s in _specs(case)]
        self.case, self.dim = case, case["dim"]
        d = self.dim
        T = lambda v: torch.tensor(v, dtype=F64, device=DEV)  # noqa: E731
        starts = []
        with tempfile.TemporaryDirectory() as wd:
            for k, s in enumerate(full):
                # the lattice, its colloid shells and ids are inputs: the engine's start
                starts.append(sph_b200.host_setup(
                    sph_input.write_input(os.path.join(wd, "input_%d" % k), **s))[0])
        n = [len(a["x"]) for a in starts]
        nb = len(full)
        self.box = torch.repeat_interleave(torch.arange(nb, device=DEV), torch.tensor(n, device=DEV))
        cat = lambda q: torch.from_numpy(np.concatenate([a[q] for a in starts])).to(DEV)  # noqa: E731
        self.type = cat("type").long()
        self.m = cat("mass")
        self.fluid = self.type == 0
        start = _disorder(full, seed, self.fluid, self.box, [cat(q) for q in "xyz"[:d]])
        self.x = torch.stack([start[q] for q in "xyz"[:d]])
        self.v = torch.stack([start["v" + q] for q in "xyz"[:d]])
        names = ["cxx", "cxy", "cyy", "cxz", "cyz", "czz"][:3 if d == 2 else 6]
        self.cnames = names
        self.c = torch.stack([torch.where(self.fluid, start[q], cat(q)) for q in names])
        # box constants
        B = {}
        B["L"] = T([s["L"] for s in full]).T.contiguous()
        for q in ("dt", "t0", "eta", "zeta", "tau", "rho", "c", "P0", "Vwall_bottom", "Vwall_top",
                  "coll_R", "coll_rho", "F0_repulsion", "tau_repulsion", "F0_magnetic",
                  "omega_magnetic", "coll_repulsion_cuton", "cutoff_magnetic"):
            B[q] = T([float(s[q]) for s in full])
        rcut = T([s["L"][0] / s["N"][0] * s["overlap"] for s in full])
        B["rcut"] = rcut
        B["cw"] = 63.0 / (478.0 * math.pi * rcut ** 2) if d == 2 else 27.0 / (120.0 * math.pi * rcut ** 3)
        B["nkT"] = T([s["np"] * s["kT"] for s in full])
        B["a"] = 5.0 * B["eta"] / 3.0 - B["zeta"]
        B["b"] = (5.0 if d == 3 else 4.0) * (B["zeta"] + B["eta"] / 3.0)
        self.B = B
        self.wall = bool(full[0]["wall"])
        self.periodic = [True, not self.wall, True][:d]
        self.ext = (full[0]["ext_force_type"], [float(f) for f in full[0]["ext_force"]])
        # colloids
        self.coll_moves = [s["coll_move"] == 0 for s in full]
        centres, cbox = [], []
        for k, s in enumerate(full):
            for xc in s["coll_x"]:
                centres.append(list(xc)[:d])
                cbox.append(k)
        self.nc = len(centres)
        if self.nc:
            self.cbox = torch.tensor(cbox, device=DEV)
            first = torch.searchsorted(self.cbox, torch.arange(nb, device=DEV))
            self.X = T(centres).T.contiguous()
            self.V = torch.zeros_like(self.X)
            z = torch.zeros(self.nc, dtype=F64, device=DEV)
            self.om = torch.zeros(3, self.nc, dtype=F64, device=DEV)
            self.theta = z.clone()
            self.q = torch.stack([z + 1.0, z, z, z])
            self.shell = torch.nonzero(self.type >= 3).flatten()
            self.owner = first[self.box[self.shell]] + self.type[self.shell] - 3
            self.body = self._image(self.x0(cat)[:, self.shell] - self.X[:, self.owner],
                                    self.box[self.shell])
            self.moving = torch.tensor(self.coll_moves, device=DEV)[self.cbox]
            R, rho = B["coll_R"][self.cbox], B["coll_rho"][self.cbox]
            self.M = math.pi * R ** 2 * rho if d == 2 else 4.0 / 3.0 * math.pi * R ** 3 * rho
            self.I = (0.5 if d == 2 else 0.4) * self.M * R ** 2
            full_owner = torch.full_like(self.type, -1)
            full_owner[self.shell] = self.owner
            self.owner_all = full_owner
        self.step_no = 0
        self.forces()

    def x0(self, cat):
        return torch.stack([cat(q) for q in "xyz"[:self.dim]])

    def _image(self, r, box):
        """Minimum image of separations along the periodic axes."""
        r = list(r)
        for k in range(self.dim):
            if self.periodic[k]:
                L = self.B["L"][k][box]
                r[k] = torch.where(r[k] > 0.5 * L, r[k] - L, r[k])
                r[k] = torch.where(r[k] < -0.5 * L, r[k] + L, r[k])
        return torch.stack(r)

    def _wrap(self, x, box):
        for k in range(self.dim):
            if self.periodic[k]:
                L = self.B["L"][k][box]
                x[k] = torch.where(x[k] < 0, x[k] + L, x[k])
                x[k] = torch.where(x[k] > L, x[k] - L, x[k])

    def pairs(self):
        """All ordered pairs (i, j), i != j, inside the cutoff, in chunks of int32."""
        d, B = self.dim, self.B
        width = torch.zeros_like(B["rcut"])
        if self.wall:
            width = B["rcut"]  # wall layers one cutoff thick (whole overlaps)
        span = [B["L"][k] + (2.0 * width if k == 1 else 0.0) for k in range(d)]
        nc = [torch.clamp((s / B["rcut"]).floor(), min=3).long() for s in span]
        cells = nc[0] * nc[1] * (nc[2] if d == 3 else 1)
        base = torch.cumsum(cells, 0) - cells
        idx = []
        for k in range(d):
            o = width[self.box] if k == 1 else 0.0
            ck = ((self.x[k] + o) / (span[k] / nc[k])[self.box]).floor().long()
            idx.append(torch.minimum(torch.clamp(ck, min=0), nc[k][self.box] - 1))
        n = [q[self.box] for q in nc]

        def linear(i):
            c = i[0] + n[0] * i[1]
            return base[self.box] + (c + n[0] * n[1] * i[2] if d == 3 else c)

        own = linear(idx)
        order = torch.argsort(own)
        count = torch.bincount(own, minlength=int(cells.sum()))
        begin = torch.cumsum(count, 0) - count
        out = []
        for o in range(3 ** d):
            move = [o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1][:d]
            there, ok = [], torch.ones_like(self.fluid)
            for k in range(d):
                t = idx[k] + move[k]
                if self.periodic[k]:
                    t = t % n[k]
                else:
                    ok = ok & (t >= 0) & (t < n[k])
                    t = torch.minimum(torch.clamp(t, min=0), n[k] - 1)
                there.append(t)
            cell = linear(there)
            num = torch.where(ok, count[cell], torch.zeros_like(cell))
            ends = torch.cumsum(num, 0)
            lo = 0
            total = int(ends[-1])
            done = 0
            while done < total:
                hi = int(torch.searchsorted(ends, torch.tensor(done + self.CHUNK, device=DEV), right=True))
                hi = max(hi, lo + 1)
                nn = num[lo:hi]
                i = torch.repeat_interleave(torch.arange(lo, hi, device=DEV), nn)
                at = torch.arange(i.numel(), device=DEV) + done - (ends[lo:hi] - nn)[i - lo]
                j = order[begin[cell[i]] + at]
                r = self._image(self.x[:, i] - self.x[:, j], self.box[i])
                near = ((r * r).sum(0) < (B["rcut"] ** 2)[self.box[i]]) & (i != j)
                out.append((i[near].int(), j[near].int()))
                done = int(ends[hi - 1])
                lo = hi
        return out

    def forces(self):
        d, B, box = self.dim, self.B, self.box
        pairs = self.pairs()
        N = box.numel()
        zero = lambda *s: torch.zeros(*s, N, dtype=F64, device=DEV)  # noqa: E731
        dens = B["cw"][box] * (243.0 - 6.0 * 32.0 + 15.0)  # the particle itself, W(0)
        for i, j in pairs:
            i, j = i.long(), j.long()
            r = self._image(self.x[:, i] - self.x[:, j], box[i]).norm(dim=0)
            q = 3.0 * r / B["rcut"][box[i]]
            w = (3.0 - q) ** 5 - 6.0 * torch.clamp(2.0 - q, min=0) ** 5 + 15.0 * torch.clamp(1.0 - q, min=0) ** 5
            dens.index_add_(0, i, B["cw"][box[i]] * w)
        press = (B["c"] ** 2)[box] * (self.m * dens - (B["P0"] * B["rho"])[box])
        nkT = B["nkT"][box]
        f = zero(d)
        g = zero(d, d)
        for i, j in pairs:
            i, j = i.long(), j.long()
            b = box[i]
            rv = self._image(self.x[:, i] - self.x[:, j], b)
            r = rv.norm(dim=0)
            e = rv / r
            q = 3.0 * r / B["rcut"][b]
            gw = (3.0 - q) ** 4 - 6.0 * torch.clamp(2.0 - q, min=0) ** 4 + 15.0 * torch.clamp(1.0 - q, min=0) ** 4
            gw = gw * (-15.0 * B["cw"] / B["rcut"])[b]
            fi, fj = self.fluid[i], self.fluid[j]
            v = self.v[:, i] - self.v[:, j]
            mixed = torch.nonzero(fi != fj).flatten()
            if mixed.numel():
                v[:, mixed] = self._ghost(i[mixed], j[mixed], rv[:, mixed])
            solid = (~fi) & (~fj)
            # gradient: pairs with a fluid particle (two colloids close to one another touch
            # only the gradient of their own particles, which no output holds)
            s = torch.where(solid, torch.zeros_like(gw), -gw / dens[i])
            for a in range(d):
                for c in range(d):
                    g[a, c].index_add_(0, i, s * e[a] * v[c])
            # forces: pairs with a fluid particle
            act = (~solid).to(F64)
            k = torch.where(fi, i, j)  # density (and, where i is solid, stress) of this one
            di = torch.where(fi & fj, dens[i], dens[k])
            dj = torch.where(fi & fj, dens[j], dens[k])
            ev = (e * v).sum(0)
            aux = gw / (di * dj * r)
            cj = self.c[:, j]
            ci = self.c[:, i]
            pj = torch.where(fj, press[j], press[i])
            pi = torch.where(fi, press[i], press[j])
            for a in range(d):
                t = torch.zeros_like(gw)
                for c in range(d):
                    diag = 1.0 if a == c else 0.0
                    Pj = (diag * pj - nkT[j] * _sym(cj, a, c)) / dj ** 2
                    Pi = (diag * pi - nkT[i] * _sym(ci, a, c)) / di ** 2
                    Pi = torch.where(fi, Pi, Pj)  # a solid takes its fluid partner's stress
                    t = t + (Pi + Pj) * e[c]
                t = -gw * t + B["a"][b] * aux * v[a] + B["b"][b] * aux * ev * e[a]
                f[a].index_add_(0, i, act * t)
        kind, amp = self.ext
        if kind:
            mf = torch.where(self.fluid, self.m, torch.zeros_like(self.m))
            if kind == 1:
                for a in range(d):
                    f[a] += mf * amp[a]
            elif kind == 2:
                f[0] += mf * amp[0] * torch.sin(2.0 * math.pi / B["L"][1][box] * self.x[1])
            else:
                f[0] += torch.where(self.x[1] < 0.5 * B["L"][1][box], mf * amp[0], -mf * amp[0])
        self.f, self.g, self.dens, self.press = f, g, dens, press
        rate = []
        for q in self.cnames:
            a, b_ = "xyz".index(q[1]), "xyz".index(q[2])
            t = torch.zeros_like(dens)
            for k in range(d):
                t = t + _sym(self.c, a, k) * g[k, b_] + _sym(self.c, b_, k) * g[k, a]
            t = t + ((1.0 if a == b_ else 0.0) - _sym(self.c, a, b_)) / B["tau"][box]
            rate.append(torch.where(self.fluid, t, torch.zeros_like(t)))
        self.dcdt = torch.stack(rate)
        if self.nc:
            self._colloid_forces()

    def _ghost(self, i, j, r):
        """Morris velocity difference of pairs of a fluid particle and a wall or colloid one."""
        d, B = self.dim, self.B
        first = self.fluid[i]
        fl, so = torch.where(first, i, j), torch.where(first, j, i)
        sign = torch.where(first, 1.0, -1.0)
        rf = r * sign  # from the solid particle to the fluid one
        b, t = self.box[fl], self.type[so]
        top = B["L"][1][b]
        bottom_wall = t == 1
        dist_f = torch.where(bottom_wall, self.x[1, fl], top - self.x[1, fl])
        dist_s = torch.where(bottom_wall, -self.x[1, so], self.x[1, so] - top)
        wall_v = torch.zeros(d, i.numel(), dtype=F64, device=DEV)
        wall_v[0] = torch.where(bottom_wall, B["Vwall_bottom"][b], B["Vwall_top"][b])
        rel = self.v[:, fl] - wall_v
        beta = torch.clamp(1.0 + dist_s / dist_f, max=1.5)
        out = torch.where(dist_f > 0, beta, torch.ones_like(beta)) * rel
        if self.nc:
            is_c = torch.nonzero(t >= 3).flatten()
            if is_c.numel():
                fl, so, b, rf = fl[is_c], so[is_c], b[is_c], rf[:, is_c]
                o = self.owner_all[so]
                rc = self._image(self.x[:, fl] - self.X[:, o], b)
                dc = rc.norm(dim=0)
                R = B["coll_R"][b]
                n = rc / dc
                surf = n * R
                om = self.om[:, o]
                if d == 2:
                    spin = torch.stack([-om[2] * surf[1], om[2] * surf[0]])
                else:
                    spin = torch.linalg.cross(om, surf, dim=0)
                dis = dc - R
                beta = torch.clamp(1.0 + ((rf * n).sum(0) - dis) / dis, max=1.5)
                rel = self.v[:, fl] - self.V[:, o]
                out[:, is_c] = torch.where(dis < 0, rel, beta * (rel - spin))
        return out * sign

    def _colloid_forces(self):
        d, B = self.dim, self.B
        F = torch.zeros(3, self.nc, dtype=F64, device=DEV)
        Tq = torch.zeros(3, self.nc, dtype=F64, device=DEV)
        fs = torch.zeros(3, self.shell.numel(), dtype=F64, device=DEV)
        fs[:d] = self.f[:, self.shell]
        r = torch.zeros_like(fs)
        r[:d] = self._image(self.x[:, self.shell] - self.X[:, self.owner], self.box[self.shell])
        F.index_add_(1, self.owner, fs)
        Tq.index_add_(1, self.owner, torch.linalg.cross(r, fs, dim=0))
        cb = self.cbox
        time = B["t0"] + B["dt"] * self.step_no
        ang = (B["omega_magnetic"] * time)[cb]
        mag = torch.stack([torch.cos(ang), torch.sin(ang), torch.zeros_like(ang)])
        i, j = torch.nonzero((cb[:, None] == cb[None, :]) & ~torch.eye(self.nc, dtype=torch.bool, device=DEV),
                             as_tuple=True)
        if i.numel():
            b = cb[i]
            rv = torch.zeros(3, i.numel(), dtype=F64, device=DEV)
            rv[:d] = self._image(self.X[:, i] - self.X[:, j], b)
            r2 = (rv * rv).sum(0)
            R, tr = B["coll_R"][b], B["tau_repulsion"][b]
            on, off = 2.0 * R + B["coll_repulsion_cuton"][b], 2.0 * R + 5.0 * R / tr
            c2 = torch.maximum(r2, on * on)
            rr = torch.sqrt(c2)
            ex = torch.exp(-tr * (rr - 2.0 * R) / R)
            Fm = B["F0_repulsion"][b] * tr * ex / (1.0 - ex)
            rep = torch.where(c2 <= off * off, Fm / rr, torch.zeros_like(rr)) * rv
            rm = torch.sqrt(r2) / (R if d == 3 else 1.0)
            e = rv / rm
            mi = mag[:, i]
            me = (mi * e).sum(0)
            dip = B["F0_magnetic"][b] / r2 ** 2 * (2.0 * me * mi - (5.0 * me * me - 1.0) * e)
            dip = torch.where(r2 <= (B["cutoff_magnetic"][b]) ** 2, dip, torch.zeros_like(dip))
            F.index_add_(1, i, rep + dip)
        if d == 2:
            F[2] = 0.0
            Tq[:2] = 0.0
        self.F, self.Tq = F, Tq

    def half_kick(self):
        dt = self.B["dt"][self.box]
        self.v = torch.where(self.fluid, self.v + 0.5 * dt / self.m * self.f, self.v)
        self.c = torch.where(self.fluid, self.c + 0.5 * dt * self.dcdt, self.c)
        if self.nc:
            h = 0.5 * self.B["dt"][self.cbox]
            self.V = torch.where(self.moving, self.V + h / self.M * self.F[:self.dim], self.V)
            self.om = torch.where(self.moving, self.om + h / self.I * self.Tq, self.om)

    def step(self):
        B, d = self.B, self.dim
        self.half_kick()
        dt = B["dt"][self.box]
        for t, q in ((1, "Vwall_bottom"), (2, "Vwall_top")):
            w = self.type == t
            self.v[0] = torch.where(w, B[q][self.box], self.v[0])
            self.v[1:, w] = 0.0
        free = self.type <= 2
        self.x = torch.where(free, self.x + self.v * dt, self.x)
        if self.nc:
            cdt = B["dt"][self.cbox]
            X = torch.where(self.moving, self.X + self.V * cdt, self.X)
            self._wrap(X, self.cbox)
            self.X = X
            if d == 2:
                self.theta = torch.where(self.moving, self.theta + self.om[2] * cdt, self.theta)
                c, s = torch.cos(self.theta)[self.owner], torch.sin(self.theta)[self.owner]
                p = torch.stack([self.body[0] * c - self.body[1] * s, self.body[0] * s + self.body[1] * c])
            else:
                w = self.om.norm(dim=0)
                half = 0.5 * w * cdt
                dq = torch.cat([torch.cos(half)[None], torch.sin(half) * self.om / w])
                self.q = torch.where(self.moving, _hamilton(dq, self.q), self.q)
                q = self.q[:, self.owner]
                conj = torch.cat([q[:1], -q[1:]])
                pt = torch.cat([torch.zeros_like(self.body[:1]), self.body])
                p = _hamilton(_hamilton(q, pt), conj)[1:]
            at = p + self.X[:, self.owner]
            self.x[:, self.shell] = torch.where(self.moving[self.owner], at, self.x[:, self.shell])
        self._wrap(self.x, self.box)
        self.step_no += 1
        self.forces()
        self.half_kick()

    def walls(self):
        out = []
        for t in (1, 2):
            w = torch.zeros(self.dim, self.B["dt"].numel(), dtype=F64, device=DEV)
            w.index_add_(1, self.box, torch.where(self.type == t, self.f, torch.zeros_like(self.f)))
            out.append(w.T)
        return torch.stack(out, dim=1)

    def energy(self):
        out = torch.zeros(self.B["dt"].numel(), dtype=F64, device=DEV)
        return out.index_add_(0, self.box, 0.5 * self.m * (self.v * self.v).sum(0))

    def state(self):
        d, out = self.dim, {}
        if self.nc:
            rows = list(self.X) + list(self.V)
            if d == 2:
                rows += [self.om[2], self.theta, self.F[0], self.F[1], self.Tq[2]]
            else:
                rows += list(self.om) + list(self.q) + list(self.F) + list(self.Tq)
            out["colloids"] = torch.stack(rows)
        if self.wall:
            out["walls"] = self.walls()
        fields = {q: self.x[k] for k, q in enumerate("xyz"[:d])}
        fields.update({"v" + q: self.v[k] for k, q in enumerate("xyz"[:d])})
        fields.update(dict(zip(self.cnames, self.c)))
        fields.update({"f" + q: self.f[k] for k, q in enumerate("xyz"[:d])})
        fields["dens"] = self.dens
        if self.case["kind"] == "methods":
            fields["press"] = self.press
            # the gradient next to a wall is taken for wall particles too
            fields.update({"g%s%s" % ("xyz"[a], "xyz"[b]): self.g[a, b]
                           for a in range(d) for b in range(d)})
        out["fields"] = fields
        return out


def _hamilton(a, b):
    return torch.stack([a[0] * b[0] - a[1] * b[1] - a[2] * b[2] - a[3] * b[3],
                        a[0] * b[1] + a[1] * b[0] + a[2] * b[3] - a[3] * b[2],
                        a[0] * b[2] - a[1] * b[3] + a[2] * b[0] + a[3] * b[1],
                        a[0] * b[3] + a[1] * b[2] - a[2] * b[1] + a[3] * b[0]])


def exact(case, seed):
    if case["kind"] in ("steps", "methods"):
        s = _Exact(case, seed)
        walls, energy = [], []
        for _ in range(case["steps"]):
            s.step()
            walls.append(s.walls() if s.wall else None)
            energy.append(s.energy())
        out = s.state()
        if case["kind"] == "methods":
            out["wall_series"] = torch.stack(walls)
            out["energy_series"] = torch.stack(energy)
            if case["precision"] == "fp64":
                out["cells"] = {"particle_cell": None, "particle_index": None}
        return out
    params, x, y = _network(case, seed)
    I, H, O = sph_surrogate.IN, sph_surrogate.HID, sph_surrogate.OUT
    p = params.to(DEV, F64).requires_grad_(case["kind"] == "train")
    x, y = x.to(DEV, F64), y.to(DEV, F64)

    def forward(x):
        o, h = 0, x.expand(case["heads"], -1, -1)
        for k, (rows, cols) in enumerate(((H, I), (H, H), (H, H), (O, H))):
            w = p[:, o:o + rows * cols].reshape(-1, rows, cols)
            b = p[:, o + rows * cols:o + rows * cols + rows]
            o += rows * cols + rows
            h = h @ w.transpose(1, 2) + b[:, None]
            if k < 3:
                h = torch.nn.functional.gelu(h)
        return h

    if case["kind"] == "predict":
        return forward(x)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for k, (xb, yb) in enumerate(zip(x.split(case["batch"]), y.split(case["batch"]))):
        loss = ((forward(xb) - yb) ** 2).mean(dim=(1, 2)).sum()
        g, = torch.autograd.grad(loss, p)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p = p - 1e-3 * (m / (1 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
        p.requires_grad_(True)
    return p.detach()
