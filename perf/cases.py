"""Measured cases: what a user of this package has the GPU do, through its public API.

Kinds of case (every size is a plain number of the case, every value comes from the seed):

solve     FDTDSolver: reset, load an initial pressure field, run_steps, read the probe
          traces and the four fields.  Grid edges 48..400 cells (the served stream's
          smallest edge to the large enclosure), any nz, uniform or stretched spacing, free
          field, rigid spheres and boxes or the ported enclosure, PML 8..16, and a block of a
          1- or 2-pole Debye or a Lorentz material.
room      the same loop with the features that act between steps: first-order absorbing
          planes, a membrane source, an omnidirectional and a cardioid microphone.
batch     BatchedSolver over uneven grids (edges 64..192, own step counts, spheres and boxes,
          a Debye block in each).
gradient  DifferentiableSolver: probe loss and its backward pass (density field, and the
          occupancy field where the case has one) in double-word, FP32 or FP64.
voxel     an SDF/CSG solid to a mask on the GPU: the ported enclosure, or a block with
          Helmholtz resonators cut into it.

exact() steps the same schemes with plain torch in 64 bits.
"""
import math

import numpy as np
import torch

import strata_fdtd_gb300 as sf

C, RHO, RES, COURANT = 343.0, 1.204, 1e-3, 0.5
PML_ORDER, PML_TARGET = 3, 1e-6
LARGEST = 400**3 * 400  # cell-updates of the largest listed solve


def listed():
    return [
        # the smallest request of a served stream: latency and launches
        solve("solve_small", 52, 44, 48, steps=250, pml=8),
        # the README quick start (half its steps)
        solve("quick_start_100", 100, 100, 100, steps=500, pml=10),
        # a room with obstacles on odd sizes: nz is not a multiple of the vector width
        solve("ragged_walls", 203, 167, 181, steps=200, pml=8, geometry="shapes", probes=2),
        # the large single solve: ported enclosure, 8 probes; state far larger than L2
        solve("enclosure_400", 400, 400, 400, steps=400, pml=16, geometry="enclosure", probes=8),
        # an absorber block of a 2-pole Debye material in a medium grid
        solve("absorber_debye", 176, 152, 144, steps=200, pml=8, geometry="shapes", probes=2,
              material="debye2", block=44),
        # a stretched grid around a source, with obstacles
        solve("stretched_grid", 144, 120, 132, steps=200, pml=10, geometry="shapes", probes=2,
              stretch=1.01),
        # a small room measured with microphones: work between the steps
        dict(name="room_microphones", kind="room", nx=112, ny=96, nz=120, steps=150),
        # a parameter sweep over uneven grids in one run
        dict(name="batch_uneven", kind="batch", grids=16, low=64, high=192, steps_low=60,
             steps_high=200, draw=1),
        # topology optimisation step, the default precision, full-size design grid
        gradient("gradient_dw_128", 128, 128, 128, steps=200, every=100, dtype="dw"),
        # a quick FP32 design iteration with a geometry field, odd sizes
        gradient("gradient_f32_odd", 75, 66, 61, steps=150, every=50, dtype="f32", occupancy=True),
        # geometry of the large solve
        dict(name="voxel_enclosure_400", kind="voxel", nx=400, ny=400, nz=400, shape="enclosure",
             resonators=0),
        # a served request's geometry: an absorber block with a resonator array
        dict(name="voxel_helmholtz", kind="voxel", nx=180, ny=240, nz=157, shape="helmholtz",
             resonators=16),
    ]


def solve(name, nx, ny, nz, steps, pml, geometry="free", probes=1, material="none", block=0,
          stretch=1.0):
    return dict(name=name, kind="solve", nx=nx, ny=ny, nz=nz, steps=steps, pml=pml,
                geometry=geometry, probes=probes, material=material, block=block, stretch=stretch)


def gradient(name, nx, ny, nz, steps, every, dtype, occupancy=False):
    return dict(name=name, kind="gradient", nx=nx, ny=ny, nz=nz, steps=steps, every=every,
                dtype=dtype, occupancy=occupancy)


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "room", "batch", "gradient", "voxel"])
    if kind == "solve":
        n = [log_int(rng, 48, 400) for _ in range(3)]
        c = solve("", *n, steps=0, pml=rng.randint(8, 16),
                  geometry=rng.choice(["free", "shapes", "shapes"]), probes=rng.randint(1, 8))
        style = rng.choice(["plain", "plain", "material", "stretch"])
        if style == "material":
            c["material"] = rng.choice(["debye1", "debye2", "lorentz"])
            c["block"] = rng.randint(8, max(8, min(n) - 2 * c["pml"] - 4))
        if style == "stretch":
            c["stretch"] = rng.choice([1.005, 1.01, 1.02])
        c["steps"] = min(log_int(rng, 40, 1000), max(40, LARGEST // (2 * n[0] * n[1] * n[2])))
    elif kind == "room":
        c = dict(kind="room", nx=log_int(rng, 48, 200), ny=log_int(rng, 48, 200),
                 nz=log_int(rng, 48, 200), steps=log_int(rng, 40, 400))
    elif kind == "batch":
        low = rng.randint(48, 80)
        c = dict(kind="batch", grids=rng.randint(4, 24), low=low, high=rng.randint(120, 192),
                 steps_low=rng.randint(40, 80), steps_high=rng.randint(100, 200),
                 draw=rng.randint(0, 10**6))
    elif kind == "gradient":
        n = [log_int(rng, 40, 128) for _ in range(3)]
        c = gradient("", *n, steps=rng.randint(60, 200), every=rng.choice([25, 50, 100]),
                     dtype=rng.choice(["dw", "dw", "f32", "f32", "f64"]),
                     occupancy=rng.random() < 0.5)
    else:
        shape = rng.choice(["enclosure", "helmholtz"])
        n = [log_int(rng, 100, 400) for _ in range(3)]
        c = dict(kind="voxel", nx=n[0], ny=n[1], nz=n[2], shape=shape,
                 resonators=rng.randint(4, 32) if shape == "helmholtz" else 0)
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- inputs from the seed
def shape_of(c):
    return c["nx"], c["ny"], c["nz"]


def initial_pressure(shape, rng, device):
    """A smooth pressure field, nonzero everywhere: a sum of products of cosines."""
    total = torch.zeros(shape, dtype=torch.float32, device=device)
    for _ in range(3):
        f = []
        for n in shape:
            x = torch.arange(n, dtype=torch.float64, device=device) / n
            f.append((0.55 + 0.45 * torch.cos(2 * math.pi * (rng.uniform(0.5, 4.0) * x
                                                             + rng.uniform()))).float())
        total += float(rng.uniform(0.2, 1.0)) * (f[0][:, None, None] * f[1][None, :, None]
                                                 * f[2][None, None, :])
    return total


def pinned(t):
    """A host copy in page-locked memory, as NumPy."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def shapes_mask(shape, rng):
    """1-6 rigid spheres or boxes; True = air."""
    air = np.ones(shape, dtype=bool)
    for _ in range(int(rng.integers(1, 7))):
        r = int(rng.integers(4, max(5, min(shape) // 6)))
        cen = [int(rng.integers(r, n - r)) for n in shape]
        box = tuple(slice(c - r, c + r + 1) for c in cen)
        if rng.random() < 0.5:
            i, j, k = np.ogrid[box]
            air[box] &= (i - cen[0])**2 + (j - cen[1])**2 + (k - cen[2])**2 > r * r
        else:
            air[box] = False
    return air


def air_cell(air, shape, margin, rng):
    for _ in range(10000):
        c = tuple(int(rng.integers(margin, n - margin)) for n in shape)
        if air is None or air[c]:
            return c
    return tuple(int(v) for v in np.argwhere(air)[0])


ENCLOSURE = dict(outer=(0.2, 0.12, 0.3), inner=(0.176, 0.096, 0.276), radius=0.025, port=0.08)


def enclosure_solid(extent):
    """Box enclosure with a port, centred and scaled to the grid (of extent 0.4 m: as it is)."""
    s = min(extent) / 0.4
    cen = tuple(e / 2 for e in extent)
    z0 = cen[2] - 0.5 * ENCLOSURE["outer"][2] * s
    return sf.Difference(
        sf.Box(center=cen, size=tuple(v * s for v in ENCLOSURE["outer"])),
        sf.Box(center=cen, size=tuple(v * s for v in ENCLOSURE["inner"])),
        sf.Cylinder(p1=(cen[0], cen[1], z0), p2=(cen[0], cen[1], z0 + ENCLOSURE["port"] * s),
                    radius=ENCLOSURE["radius"] * s))


def enclosure_air(shape, device):
    """The complement of enclosure_solid on a uniform grid, from its definition."""
    ext = [n * RES for n in shape]
    s = min(ext) / 0.4
    x, y, z = (torch.arange(n, dtype=torch.float64, device=device) * RES + RES / 2 - e / 2
               for n, e in zip(shape, ext))
    x, y, z = x[:, None, None], y[None, :, None], z[None, None, :]

    def box(size):
        return ((x.abs() <= size[0] * s / 2) & (y.abs() <= size[1] * s / 2)
                & (z.abs() <= size[2] * s / 2))

    z0 = -0.5 * ENCLOSURE["outer"][2] * s
    port = ((x**2 + y**2 <= (ENCLOSURE["radius"] * s)**2) & (z >= z0)
            & (z <= z0 + ENCLOSURE["port"] * s))
    return ~(box(ENCLOSURE["outer"]) & ~box(ENCLOSURE["inner"]) & ~port)


def resonator_block(shape, count, rng):
    """A solid block on the low-x side with resonators cut into its face."""
    cav, neck = int(rng.integers(10, 21)), int(rng.integers(3, 9))
    lo, hi = 10, [n - 10 for n in shape]
    per = math.ceil(math.sqrt(count))
    cut = []
    for q in range(count):
        cy = lo + (q % per + 0.5) * (hi[1] - lo) / per
        cz = lo + (q // per + 0.5) * (hi[2] - lo) / per
        cut.append(sf.HelmholtzResonator(
            position=((lo + cav / 2 + 2) * RES, cy * RES, cz * RES), cavity_shape="box",
            cavity_size=(cav * RES,) * 3, neck_length=4 * RES, neck_radius=neck * RES,
            neck_direction=(1, 0, 0)))
    block = sf.Box(min_corner=(lo * RES,) * 3,
                   max_corner=((lo + cav + 6) * RES, hi[1] * RES, hi[2] * RES))
    return sf.Difference(block, sf.Union(*cut))


def material_poles(style, rng):
    """[(kind, target, strength, tau | omega_0, gamma)] of a material that the scheme steps
    stably."""
    out = []
    if style == "lorentz":
        f0 = float(rng.uniform(800.0, 3000.0))
        out.append(("lorentz", "density", float(rng.uniform(0.05, 0.2)), 2 * math.pi * f0,
                    float(rng.uniform(500.0, 2000.0))))
    else:
        for target in ("density", "modulus")[:int(style[-1])]:
            out.append(("debye", target, float(rng.uniform(0.1, 0.3)),
                        float(np.exp(rng.uniform(np.log(2e-4), np.log(1e-3)))), 0.0))
    return out


class Setup:
    """Everything one solve is made from, drawn from the seed."""

    def __init__(self, c, seed, device):
        rng = np.random.default_rng(seed)
        self.shape = shape_of(c)
        self.pml, self.steps, self.stretch = c["pml"], c["steps"], c["stretch"]
        self.air = None
        self.enclosure = c["geometry"] == "enclosure"
        if self.enclosure:
            self.air = enclosure_air(self.shape, device).cpu().numpy()
        elif c["geometry"] == "shapes":
            self.air = shapes_mask(self.shape, rng)
        self.poles, self.box = [], None
        if c["material"] != "none":
            self.poles = material_poles(c["material"], rng)
            b = min(c["block"], min(self.shape) - 2 * self.pml - 2)
            lo = [int(rng.integers(self.pml, n - self.pml - b)) for n in self.shape]
            self.box = [(v, v + b) for v in lo]
        self.source = air_cell(self.air, self.shape, self.pml, rng)
        self.frequency = float(rng.uniform(2000.0, 8000.0))
        self.probes = [air_cell(self.air, self.shape, self.pml, rng) for _ in range(c["probes"])]
        self.p0 = initial_pressure(self.shape, rng, device)

    def grid(self):
        if self.stretch == 1.0:
            return sf.UniformGrid(self.shape, RES)
        return sf.NonuniformGrid(*(axis_of(n, self.stretch)[0] for n in self.shape))

    def solver(self):
        s = sf.FDTDSolver(grid=self.grid(), c=C, rho=RHO, courant=COURANT)
        s.add_boundary(sf.PML(depth=self.pml))
        if self.enclosure:
            s.set_geometry_sdf(enclosure_solid([n * RES for n in self.shape]))
        elif self.air is not None:
            s.set_geometry(self.air)
        if self.poles:
            mat = sf.SimpleMaterial(name="block", _rho=RHO, _c=C, _poles=[
                sf.Pole(sf.PoleType.DEBYE, delta_chi=x, target=t, tau=a) if k == "debye" else
                sf.Pole(sf.PoleType.LORENTZ, delta_chi=x, target=t, omega_0=a, gamma=g)
                for k, t, x, a, g in self.poles])
            s.set_material_box(s.register_material(mat), *self.box)
        s.add_source(sf.GaussianPulse(position=self.source, frequency=self.frequency))
        for q, pos in enumerate(self.probes):
            s.add_probe("p%d" % q, pos)
        return s


def uneven(c):
    """The members of a batch case: shapes and step counts, fixed by the case alone."""
    rng = np.random.default_rng(c["draw"])
    out = []
    for _ in range(c["grids"]):
        n = [int(round(math.exp(rng.uniform(math.log(c["low"]), math.log(c["high"])))))
             for _ in range(3)]
        out.append(solve("", *n, steps=int(rng.integers(c["steps_low"], c["steps_high"] + 1)),
                         pml=8, geometry="shapes", probes=2, material="debye2",
                         block=int(rng.integers(10, 31))))
    return out


class Room:
    """A room with absorbing planes, a loudspeaker membrane, a tone burst and microphones."""

    def __init__(self, c, seed, device):
        rng = np.random.default_rng(seed)
        self.shape, self.steps = shape_of(c), c["steps"]
        ext = [n * RES for n in self.shape]
        self.plane = int(rng.integers(4, self.shape[2] // 2))
        self.centre = (ext[0] / 2, ext[1] / 2, (self.plane + 0.5) * RES)
        self.size = (ext[0] * 0.4, ext[1] * 0.3)
        self.f_membrane, self.f_point = (float(rng.uniform(2000.0, 8000.0)) for _ in range(2))
        self.point = air_cell(None, self.shape, 8, rng)
        self.probe = air_cell(None, self.shape, 8, rng)
        self.mics = [tuple(float(rng.uniform(0.1, 0.9)) * e for e in ext) for _ in range(2)]
        d = rng.normal(size=3)
        self.direction = tuple(float(v) for v in d / np.linalg.norm(d))
        self.up = (0.0, 0.0, 1.0) if abs(self.direction[2]) < 0.9 else (1.0, 0.0, 0.0)
        self.p0 = initial_pressure(self.shape, rng, device)

    def solver(self):
        s = sf.FDTDSolver(grid=sf.UniformGrid(self.shape, RES), c=C, rho=RHO, courant=COURANT)
        s.add_boundary(sf.ABCFirstOrder())
        s.add_source(sf.RectangularMembraneSource(
            center=self.centre, normal_axis="z", size=self.size,
            waveform=sf.GaussianPulse(position=(0, 0, 0), frequency=self.f_membrane)))
        s.add_source(sf.GaussianPulse(position=self.point, frequency=self.f_point))
        s.add_probe("p0", self.probe)
        s.add_microphone(self.mics[0], name="omni")
        s.add_microphone(self.mics[1], name="cardioid", pattern="cardioid",
                         direction=self.direction, up=self.up)
        return s


class Design:
    """A design field, an optional occupancy field and a target trace."""

    def __init__(self, c, seed, device):
        rng = np.random.default_rng(seed)
        self.shape, self.steps = shape_of(c), c["steps"]
        real = torch.float32 if c["dtype"] == "f32" else torch.float64
        self.pml = max(4, min(10, min(self.shape) // 6))
        self.source = tuple(n // 2 for n in self.shape)
        off = [max(4, n // 8) for n in self.shape]
        self.probes = [(self.source[0] + off[0], self.source[1], self.source[2]),
                       (self.source[0], self.source[1] - off[1], self.source[2] + off[2])]
        self.theta = initial_pressure(self.shape, rng, device).to(real)
        self.phi = None
        if c["occupancy"]:
            f = initial_pressure(self.shape, rng, device)
            self.phi = (0.8 * f / f.max()).to(real)
            self.phi[self.source] = 0
        t = torch.arange(self.steps, dtype=torch.float64, device=device)[:, None]
        w = torch.tensor(rng.uniform(0.02, 0.2, size=(1, 2)), dtype=torch.float64, device=device)
        self.target = (0.02 * torch.sin(w * t)).to(real)
        self.frequency = float(rng.uniform(8000.0, 12000.0))


# ------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind, dev = case["kind"], torch.device("cuda")
    if kind in ("solve", "room"):
        s = (Setup if kind == "solve" else Room)(case, seed, dev)
        return dict(kind=kind, solver=s.solver(), p0=pinned(s.p0), steps=s.steps)
    if kind == "batch":
        members = [Setup(m, seed * 1000 + q, dev) for q, m in enumerate(uneven(case))]
        solvers = [m.solver() for m in members]
        return dict(kind=kind, solvers=solvers, batch=sf.BatchedSolver(solvers),
                    p0=[pinned(m.p0) for m in members], steps=[m.steps for m in members])
    if kind == "gradient":
        d = Design(case, seed, dev)
        dtype = {"dw": "dw", "f32": torch.float32, "f64": torch.float64}[case["dtype"]]
        ds = sf.DifferentiableSolver(d.shape, RES, c=C, rho0=RHO, courant=COURANT,
                                     pml_depth=d.pml, source=d.source, frequency=d.frequency,
                                     probes=d.probes, dtype=dtype, checkpoint_every=case["every"])
        return dict(kind=kind, solver=ds, theta=d.theta, phi=d.phi, target=d.target, steps=d.steps)
    shape = shape_of(case)
    rng = np.random.default_rng(seed)
    if case["shape"] == "enclosure":
        solid = enclosure_solid([n * RES for n in shape]).translate(
            tuple(float(v) for v in rng.uniform(-0.01, 0.01, size=3)))
    else:
        solid = resonator_block(shape, case["resonators"], rng)
    return dict(kind=kind, solid=solid, grid=sf.UniformGrid(shape, RES))


def run(state):
    kind = state["kind"]
    if kind in ("solve", "room"):
        s = state["solver"]
        s.reset()
        s.load_fields_async(p=state["p0"])
        s.run_steps(state["steps"])
        out = dict(s.device_fields(), traces=s.get_probe_data())
        if kind == "room":
            out["microphones"] = {n: m.get_waveform() for n, m in s.microphones.items()}
        return out
    if kind == "batch":
        for s, p0 in zip(state["solvers"], state["p0"]):
            s.reset()
            s.load_fields_async(p=p0)
        state["batch"].run_steps(state["steps"])
        out = {}
        for q, s in enumerate(state["solvers"]):
            f = s.device_fields()
            t = s.get_probe_data()
            out["m%d" % q] = [torch.cat([f[n].reshape(-1) for n in ("p", "vx", "vy", "vz")]),
                              np.stack([t["p0"], t["p1"]])]
        return out
    if kind == "gradient":
        theta = state["theta"].clone().requires_grad_()
        phi = None if state["phi"] is None else state["phi"].clone().requires_grad_()
        loss = state["solver"].loss(theta, state["target"], state["steps"], occupancy=phi)
        loss.backward()
        return dict(loss=loss.detach(), theta=theta.grad, phi=None if phi is None else phi.grad)
    return state["solid"].voxelize_device(state["grid"], invert=True)


# ------------------------------------------------------------------------------- work
def solve_work(c):
    n = c["nx"] * c["ny"] * c["nz"]
    block = c["block"]**3 if c["material"] != "none" else 0
    poles = {"none": 0, "debye1": 1, "debye2": 2, "lorentz": 1}[c["material"]]
    # per cell and step: three faces of 3 operations, 7 for the pressure, 6 decays; per pole
    # and block cell 3 for the recursion and up to 9 for the faces it corrects
    return dict(bytes=4 * n + 16 * n + (n if c["geometry"] != "free" else 0),
                flops=c["steps"] * (22 * n + 12 * poles * block))


def work(case):
    kind = case["kind"]
    if kind == "solve":
        return solve_work(case)
    n = 1
    if kind != "batch":
        n = case["nx"] * case["ny"] * case["nz"]
    if kind == "room":
        return dict(bytes=20 * n, flops=16 * n * case["steps"])
    if kind == "batch":
        w = [solve_work(m) for m in uneven(case)]
        return dict(bytes=sum(v["bytes"] for v in w), flops=sum(v["flops"] for v in w))
    if kind == "gradient":
        # fields in and gradients out; forward 22, adjoint 30 operations per cell and step
        width = 4 if case["dtype"] == "f32" else 8
        return dict(bytes=(4 if case["occupancy"] else 2) * width * n,
                    flops=52 * n * case["steps"])
    return dict(bytes=n, flops=n)


# ------------------------------------------------------------------------ 64-bit values
def pulse(f, t):
    sigma = 1.0 / (np.pi * 2.0 * f)
    t0 = 4.0 * sigma
    return float(np.exp(-((t - t0)**2) / (2 * sigma**2)) * np.sin(2 * np.pi * f * (t - t0)))


def decays(coords, widths, depth, uniform, spacing, dt, device):
    """exp(-sigma dt) of one axis: cubic profile over the layer's cells (uniform) or metres."""
    n = len(coords)
    smax = -(PML_ORDER + 1) * C * math.log(PML_TARGET) / (2 * depth * spacing)
    s = np.zeros(n)
    if uniform:
        for q in range(depth):
            s[q] = ((depth - q) / depth)**PML_ORDER
        for q in range(n - depth, n):
            s[q] = ((q - (n - depth - 1)) / depth)**PML_ORDER
    else:
        d = depth if depth < n // 2 else max(1, n // 4)
        lo_t, hi_t = widths[:d].sum(), widths[-d:].sum()
        lo_x = coords[d] - widths[d] / 2
        hi_x = coords[n - d - 1] + widths[n - d - 1] / 2
        for q in range(d):
            s[q] = min(1.0, (lo_x - coords[q]) / lo_t)**PML_ORDER
        for q in range(n - d, n):
            s[q] = min(1.0, (coords[q] - hi_x) / hi_t)**PML_ORDER
    return torch.tensor(np.exp(-smax * s * dt), dtype=torch.float64, device=device)


def axis_of(n, ratio):
    """Cell centres and widths of one axis (widths growing outward from the middle)."""
    if ratio == 1.0:
        c = np.arange(n) * RES + RES / 2
        return c, np.full(n, RES)
    w = RES * ratio**np.abs(np.arange(n) - (n - 1) / 2)
    c = np.cumsum(w) - w / 2
    width = np.empty_like(c)
    width[1:-1] = (c[2:] - c[:-2]) / 2
    width[0], width[-1] = c[1] - c[0], c[-1] - c[-2]
    return c, width


def along(v, axis):
    return v.reshape([-1 if a == axis else 1 for a in range(3)])


class Exact:
    """The staggered update in 64 bits: velocities, rigid walls, pressure, PML decays."""

    def __init__(self, shape, p0, air=None, pml=0, stretch=1.0, poles=(), box=None):
        dev = p0.device
        self.shape, self.dev = shape, dev
        axes = [axis_of(n, stretch) for n in shape]
        uniform = stretch == 1.0
        self.dx = float(min(w.min() for _, w in axes))
        self.dt = COURANT * self.dx / (C * math.sqrt(3))
        self.p = p0.double()
        self.v = [torch.zeros(shape, dtype=torch.float64, device=dev) for _ in range(3)]
        f64 = dict(dtype=torch.float64, device=dev)
        self.cv = [along(torch.tensor(-self.dt / RHO / np.diff(c), **f64), a)
                   for a, (c, _) in enumerate(axes)]
        self.inv = [along(torch.tensor(1.0 / w, **f64), a) for a, (_, w) in enumerate(axes)]
        self.cp = -RHO * C**2 * self.dt
        self.decay = None
        if pml:
            self.decay = [along(decays(c, w, pml, uniform, self.dx, self.dt, dev), a)
                          for a, (c, w) in enumerate(axes)]
        self.air, self.open = None, None
        if air is not None:
            self.air = torch.as_tensor(air, device=dev)
            self.open = [self.lo(self.air, a) & self.hi(self.air, a) for a in range(3)]
        self.poles = [dict(kind=k, target=t, J=None, **self.pole(k, x, a, g))
                      for k, t, x, a, g in poles]
        self.box = None
        if poles:
            self.box = tuple(slice(*b) for b in box)
            for q in self.poles:
                q["J"] = torch.zeros_like(self.p[self.box])
                q["old"] = torch.zeros_like(q["J"])

    def lo(self, x, a):
        return x.narrow(a, 0, x.shape[a] - 1)

    def hi(self, x, a):
        return x.narrow(a, 1, x.shape[a] - 1)

    def pole(self, kind, x, a, g):
        if kind == "debye":
            return dict(co=(a / self.dt / (1 + a / self.dt), 0.0, x / (1 + a / self.dt)))
        c = 1 + g * self.dt / 2
        return dict(co=((2 - a**2 * self.dt**2) / c, -(1 - g * self.dt / 2) / c,
                        x * a**2 * self.dt**2 / c))

    def advance(self, q, f):
        c0, c1, c2 = q["co"]
        q["J"], q["old"] = c0 * q["J"] + c1 * q["old"] + c2 * f, q["J"]

    def step(self):
        for q in self.poles:
            if q["target"] == "density":
                self.advance(q, self.p[self.box])
        for a in range(3):
            if self.shape[a] > 1:
                v = self.lo(self.v[a], a)
                v += self.cv[a] * (self.hi(self.p, a) - self.lo(self.p, a))
                for q in self.poles:
                    if q["target"] == "density":
                        self.lo(self.v[a][self.box], a).add_(
                            self.hi(q["J"], a) - self.lo(q["J"], a),
                            alpha=-self.dt / RHO / self.dx)
                if self.open is not None:
                    v *= self.open[a]
        div = 0
        for a in range(3):
            d = self.v[a].clone()
            self.hi(d, a).sub_(self.lo(self.v[a], a))
            div = div + d.mul_(self.inv[a])
        self.p += self.cp * div
        for q in self.poles:
            if q["target"] == "modulus":
                self.advance(q, div[self.box])
                self.p[self.box] += -RHO * C**2 * self.dt * q["J"]
        if self.air is not None:
            self.p *= self.air
        if self.decay is not None:
            for a in range(3):
                self.v[a] *= self.decay[a]
                self.p *= self.decay[a]


def exact_solve(setup):
    e = Exact(setup.shape, setup.p0, setup.air, setup.pml, setup.stretch, setup.poles, setup.box)
    rows, t = [], 0.0
    src_air = setup.air is None or bool(setup.air[setup.source])
    at = torch.tensor(setup.probes, device=e.dev).T
    for _ in range(setup.steps):
        e.step()
        if src_air:
            e.p[setup.source] += pulse(setup.frequency, t)
        rows.append(e.p[at[0], at[1], at[2]])
        t += e.dt
    return e, torch.stack(rows)


def corners(pos):
    base = [int(v) for v in pos]
    out = []
    for d in ((a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)):
        w = 1.0
        for q in range(3):
            f = pos[q] - base[q]
            w *= f if d[q] else 1 - f
        out.append((tuple(base[q] + d[q] for q in range(3)), w))
    return out


def sample(field, pos):
    lim = [n - 1 for n in field.shape]
    return sum(w * field[tuple(min(i, m) for i, m in zip(c, lim))] for c, w in corners(pos))


def exact_room(r):
    e = Exact(r.shape, r.p0)
    m = (C * e.dt - e.dx) / (C * e.dt + e.dx)
    prev = [[torch.zeros_like(e.p.select(a, 0)) for _ in range(2)] for a in range(3)]
    x, y = (torch.tensor(np.arange(n) * RES + RES / 2 - c, dtype=torch.float64, device=e.dev)
            for n, c in zip(r.shape[:2], r.centre[:2]))
    w = (torch.sin(math.pi * (x / r.size[0] + 0.5))[:, None]
         * torch.sin(math.pi * (y / r.size[1] + 0.5))[None, :])
    w = w * ((x.abs() <= r.size[0] / 2)[:, None] & (y.abs() <= r.size[1] / 2)[None, :])
    w = w.abs() / w.abs().max()
    g = [[v / RES for v in pos] for pos in r.mics]
    rows, t = [], 0.0
    for _ in range(r.steps):
        e.step()
        for a in range(3):
            n = r.shape[a]
            for side, (b, i) in enumerate(((0, 1), (n - 1, n - 2))):
                inner = e.p.select(a, i).clone()
                e.p.select(a, b).copy_(prev[a][side] + m * (inner - e.p.select(a, b)))
                prev[a][side] = inner
        e.p[:, :, r.plane] += pulse(r.f_membrane, t) * w
        e.p[r.point] += pulse(r.f_point, t)
        vd = 0
        for a in range(3):
            h = list(g[1])
            h[a] -= 0.5
            h = [max(0.0, min(v, n - 1.001)) for v, n in zip(h, r.shape)]
            vd = vd + r.direction[a] * sample(e.v[a], h)
        rows.append(torch.stack([e.p[r.probe], sample(e.p, g[0]),
                                 0.5 * sample(e.p, g[1]) + 0.5 * RHO * C * vd]))
        t += e.dt
    return e, torch.stack(rows)


def exact_gradient(d):
    """Loss and gradients by torch.autograd through the 64-bit scheme, segments recomputed."""
    from torch.utils.checkpoint import checkpoint

    dev, n = d.theta.device, d.shape
    dt = COURANT * RES / (C * math.sqrt(3))
    dt_dx = dt / RES
    cp = -RHO * C**2 * dt_dx
    theta = d.theta.double().requires_grad_()
    phi = None if d.phi is None else d.phi.double().requires_grad_()
    axes = [axis_of(v, 1.0) for v in n]
    dec = [along(decays(c, w, d.pml, True, RES, dt, dev), a) for a, (c, w) in enumerate(axes)]
    b = 1.0 / (RHO * (1 + theta))
    cv = []
    for a in range(3):
        f = -dt_dx * 0.5 * (b.narrow(a, 0, n[a] - 1) + b.narrow(a, 1, n[a] - 1))
        if phi is not None:
            f = f * ((1 - phi.narrow(a, 0, n[a] - 1)) * (1 - phi.narrow(a, 1, n[a] - 1)))
        cv.append(f)
    onehot = torch.zeros(n, dtype=torch.float64, device=dev)
    onehot[d.source] = 1.0
    t, values = 0.0, []
    for _ in range(d.steps):
        values.append(pulse(d.frequency, t))
        t += dt
    zero = [torch.zeros([1 if q == a else m for q, m in enumerate(n)], dtype=torch.float64,
                        device=dev) for a in range(3)]

    def segment(first, last, p, vx, vy, vz, *cv):
        v, rows = [vx, vy, vz], []
        for s in range(first, last):
            div = 0
            for a in range(3):  # faces between cells only: the last one never moves
                v[a] = v[a] + cv[a] * (p.narrow(a, 1, n[a] - 1) - p.narrow(a, 0, n[a] - 1))
                div = div + torch.cat([v[a], zero[a]], a) - torch.cat([zero[a], v[a]], a)
            p = (p + cp * div) * dec[0] * dec[1] * dec[2] + values[s] * onehot
            v = [v[a] * dec[a].narrow(a, 0, n[a] - 1) for a in range(3)]
            rows.append(torch.stack([p[q] for q in d.probes]))
        return (p, *v, torch.stack(rows))

    state = [torch.zeros(n, dtype=torch.float64, device=dev)] + [torch.zeros_like(f) for f in cv]
    traces = []
    for s in range(0, d.steps, 20):
        *state, tr = checkpoint(segment, s, min(s + 20, d.steps), *state, *cv, use_reentrant=False)
        traces.append(tr)
    loss = ((torch.cat(traces) - d.target.double())**2).sum()
    loss.backward()
    return dict(loss=loss.detach(), theta=theta.grad, phi=None if phi is None else phi.grad)


def exact(case, seed):
    kind, dev = case["kind"], torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "voxel":
        return None  # a mask: bytes
    if kind == "gradient":
        return exact_gradient(Design(case, seed, dev))
    if kind == "batch":
        out = {}
        for q, m in enumerate(uneven(case)):
            e, rows = exact_solve(Setup(m, seed * 1000 + q, dev))
            out["m%d" % q] = [torch.cat([f.reshape(-1) for f in (e.p, *e.v)]),
                              rows.T.contiguous()]
        return out
    if kind == "room":
        e, rows = exact_room(Room(case, seed, dev))
        out = dict(p=e.p, vx=e.v[0], vy=e.v[1], vz=e.v[2], traces=dict(p0=rows[:, 0]),
                   microphones=dict(omni=rows[:, 1], cardioid=rows[:, 2]))
        return out
    e, rows = exact_solve(Setup(case, seed, dev))
    return dict(p=e.p, vx=e.v[0], vy=e.v[1], vz=e.v[2],
                traces={"p%d" % q: rows[:, q] for q in range(rows.shape[1])})
