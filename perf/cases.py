"""Workloads that time this solver through its public entry points.

Each case is one call pattern of a program that uses the stepper: a solve
restarted from a host state (that reads back u, v and sigma, or with
``checkpoint`` the whole state), a time history, result frames written while the
device steps, a batched parameter sweep, a stream of served requests.  The
meshes, materials and velocities are the ones of ``workloads`` (which also
feed the tests and the benchmark), in their sizes and in odd ones.

Results of FP64 solves are taken as the float64 arrays the calls fill.  Results
of mixed solves are kept as float32, the type in which the mixed stepper holds
stresses, hourglass history and velocities; a program that stores or
post-processes a mixed solve has no use for more.
"""
import dataclasses
import math

import numpy as np
import torch

from enscdynamics_b200 import capi
from enscdynamics_b200 import serving as S
from enscdynamics_b200 import workloads as W

PRECISION = {"fp64": capi.FP64, "mixed": capi.MIXED}


def listed():
    return [
        # the parity-sized cantilever: 320 elements, elastic, FP64; latency and launches are all of its time
        dict(name="cantilever_fp64", kind="solve", precision="fp64", shape="cantilever", nx=20, ny=4, nz=4,
             plastic=False, gravity=False, cycles=2000, checkpoint=False),
        # a tip history of the same cantilever: short calls, each with its result read back, not a multiple of
        # any graph length
        dict(name="history_mixed", kind="history", precision="mixed", shape="cantilever", nx=20, ny=4, nz=4,
             plastic=False, gravity=False, cycles=50, frames=12),
        # a thin elastic plate under ramped gravity, odd cell counts, FP64: an ordinary small part
        dict(name="plate_fp64", kind="solve", precision="fp64", shape="plate", nx=83, ny=83, nz=4,
             plastic=False, gravity=True, cycles=1000, checkpoint=True),
        # a mid-sized J2 block with odd cell counts, mixed
        dict(name="midblock_mixed", kind="solve", precision="mixed", shape="block", nx=61, ny=37, nz=19,
             plastic=True, gravity=False, cycles=1000, checkpoint=False),
        # the plastic impact bar (195,840 elements): a butterfly mesh whose nodes repeat local slots
        dict(name="bar_fp64", kind="solve", precision="fp64", shape="bar", nx=24, ny=11, nz=120,
             plastic=True, gravity=False, cycles=300, checkpoint=True),
        dict(name="bar_mixed", kind="solve", precision="mixed", shape="bar", nx=24, ny=11, nz=120,
             plastic=True, gravity=False, cycles=300, checkpoint=True),
        # the large elastic-plastic block: 2,097,152 elements, end to end from host state to host results
        dict(name="block_fp64", kind="solve", precision="fp64", shape="block", nx=256, ny=128, nz=64,
             plastic=True, gravity=False, cycles=250, checkpoint=False),
        dict(name="block_mixed", kind="solve", precision="mixed", shape="block", nx=256, ny=128, nz=64,
             plastic=True, gravity=False, cycles=500, checkpoint=False),
        # result frames (x, u, v, a, reactions, sigma) taken while the next interval runs
        dict(name="output_mixed", kind="output", precision="mixed", shape="block", nx=128, ny=64, nz=32,
             plastic=True, gravity=False, cycles=250, frames=4),
        # the batched sweep: uneven cantilevers and plates, each with its own material, dt and clock
        dict(name="sweep_mixed", kind="sweep", precision="mixed", instances=48, ne_min=2000, ne_max=60000,
             cycles=750),
        dict(name="sweep_fp64", kind="sweep", precision="fp64", instances=24, ne_min=2000, ne_max=60000,
             cycles=500),
        # a burst of served requests: host preparation on threads, admission, stepping, retirement
        dict(name="serve_mixed", kind="serve", precision="mixed", instances=16, ne_min=1000, ne_max=120000,
             cycles=600),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "history", "output", "sweep", "serve"])
    precision = rng.choice(["fp64", "mixed"])
    if kind in ("sweep", "serve"):
        lo = int(round(math.exp(rng.uniform(math.log(1000), math.log(8000)))))
        hi = int(round(math.exp(rng.uniform(math.log(16000), math.log(120000)))))
        return dict(kind=kind, precision=precision if kind == "sweep" else "mixed", instances=rng.randint(3, 24),
                    ne_min=lo, ne_max=hi, cycles=rng.randint(150, 700))
    shape = rng.choice(["cantilever", "plate", "block", "bar"])
    top = 1.5e6 if kind == "solve" else 2.0e5
    target = math.exp(rng.uniform(math.log(200.0), math.log(top)))
    if shape == "cantilever":
        k = max(2, int(round((target / 5.0) ** (1.0 / 3.0))))
        nx, ny, nz = 5 * k + rng.randint(0, 3), k, k
    elif shape == "plate":
        k = max(4, int(round(math.sqrt(target / 4.0))))
        nx, ny, nz = k, k, 4
    elif shape == "block":
        k = max(2.0, (target / 8.0) ** (1.0 / 3.0))
        nx, ny, nz = int(4 * k) + rng.randint(0, 2), int(2 * k) + rng.randint(0, 2), max(2, int(k))
    else:
        k = max(2, int(round((target / 14.0) ** (1.0 / 3.0))))
        nx, ny, nz = k, max(2, k // 2), max(4, 5 * k)
    ne = nx * nx * nz + 4 * nx * ny * nz if shape == "bar" else nx * ny * nz
    # cycles: the more the smaller the mesh, never more work than the large block
    most = max(40, int(min(2000.0, 2.0e8 / ne)))
    cycles = rng.randint(max(20, most // 4), most)
    case = dict(kind=kind, precision=precision, shape=shape, nx=nx, ny=ny, nz=nz, plastic=rng.random() < 0.6,
                gravity=rng.random() < 0.3, cycles=cycles)
    if kind == "solve":
        # restart files: of FP64 solves, and of mixed ones early in a solve
        case["checkpoint"] = (precision == "fp64" or cycles <= 300) and rng.random() < 0.5
    else:
        case["frames"] = rng.randint(2, 8)
        case["cycles"] = max(8, cycles // case["frames"])
    return case


# ---- problems ----------------------------------------------------------------

AMPLITUDE = [(0.0, 0.2), (4.0e-5, 1.0), (3.0e-4, 0.4), (2.0, 0.7)]


def problem(case, seed):
    """The mesh, material, velocities and conditions of a single-solve case."""
    rng = np.random.default_rng([seed, 5])
    nx, ny, nz, plastic = case["nx"], case["ny"], case["nz"], case["plastic"]
    if case["shape"] == "block":
        p = W.block(nx, ny, nz, nx / 256.0, ny / 256.0, nz / 256.0, seed=seed, plastic=plastic)
    elif case["shape"] == "bar":
        p = W.impact_bar(nx, ny, nz, v_impact=-rng.uniform(150.0, 200.0), plastic=plastic)
    else:
        length, h = (2.0, 2.0 / nx) if case["shape"] == "cantilever" else (1.0, 1.0 / nx)
        p = W.cantilever(nx, ny, nz, length, h * ny, h * nz, vz=rng.uniform(2.0, 6.0),
                         E=rng.uniform(190e9, 220e9), yield_stress=300e6 if plastic else 0.0,
                         tangent=100e6 if plastic else 0.0)
        p.v0 *= p.mesh.x0[:, :1] / length  # bending start: from rest at the clamp to vz at the tip
        p.controls = dataclasses.replace(p.controls, factor=W.SWEEP_DT_FACTOR)
    if case["gravity"]:
        p.controls = dataclasses.replace(p.controls, gravity=(2.0e3, (0.0, 0.0, -1.0)), gravity_amplitude=AMPLITUDE)
    return p


def problems(case, seed):
    """The instances of a sweep or of a burst of requests: element counts spread evenly over the logarithm of the
    range, the same for every seed; materials and velocities from the seed.  Requests ask for uneven cycle
    counts, and half of them are elastic."""
    n = case["instances"]
    out = []
    for i in range(n):
        ne = case["ne_min"] * (case["ne_max"] / case["ne_min"]) ** (((7 * i) % n + 0.5) / n)
        p = W.sweep_instance(i, seed=seed, ne_min=ne, ne_max=ne, cycles=case["cycles"])
        if case["kind"] == "serve":
            p.cycles = case["cycles"] // 2 + (case["cycles"] * ((5 * i) % n)) // n
            if i % 4 >= 2:
                p.material = dataclasses.replace(p.material, yield_stress=0.0, tangent_modulus=0.0)
        out.append(p)
    return out


# ---- the measured passes --------------------------------------------------------

def pinned(shape):
    return torch.empty(shape, dtype=torch.float64).pin_memory()


def prepare(case, seed):
    state = {"case": case}
    prec = PRECISION[case["precision"]]
    if case["kind"] in ("sweep", "serve"):
        state["problems"] = ps = problems(case, seed)
        # room for one set of instances beside another that has just been removed
        room = dict(max_instances=len(ps), max_elements=2 * sum(p.mesh.n_elements for p in ps),
                    max_nodes=2 * sum(p.mesh.n_nodes for p in ps), budget_bytes=20 * 10 ** 9, precision=prec)
        if case["kind"] == "sweep":
            state["batch"] = capi.Batch(**room)
            state["prepared"] = [capi.Prepared(p.mesh.x0, p.mesh.conn, p.v0, material=p.material,
                                               controls=p.controls, precision=prec) for p in ps]
        else:
            state["backend"] = S.BatchBackend(fields=("u",), **room)
            state["requests"] = [W.Request(i, 0.0, p) for i, p in enumerate(ps)]
        return state
    p = problem(case, seed)
    s = capi.Stepper(p.mesh.x0, p.mesh.conn, p.v0, material=p.material, controls=p.controls, precision=prec)
    s.set_bcs(p.bc_code, p.bc_value)
    state["stepper"] = s
    state["dts"] = s.step(0)["dt_stable_min"]
    # the host program's own state and result buffers, in pinned memory
    nn, ne = s.n_nodes, s.n_elements
    shapes = {"x": (nn, 3), "u": (nn, 3), "v": (nn, 3), "sigma": (ne, 6), "qia": (ne, 12), "eps_p": (ne,)}
    keep = {k: pinned(v) for k, v in shapes.items()}
    state["host"] = {k: v.numpy() for k, v in keep.items()}
    s.download(state["host"])
    state["out"] = {k: pinned(shapes[k]) for k in (shapes if case.get("checkpoint") else ("u", "v", "sigma"))}
    state["out_np"] = {k: v.numpy() for k, v in state["out"].items()}
    state["keep"] = keep
    return state


def result(case, a):
    """A result as the program keeps it (see the module's comment)."""
    t = a if isinstance(a, torch.Tensor) else torch.from_numpy(np.asarray(a))
    return t.float() if case["precision"] == "mixed" else t


def run(state):
    case = state["case"]
    return {"solve": run_solve, "history": run_history, "output": run_output, "sweep": run_sweep,
            "serve": run_serve}[case["kind"]](case, state)


def run_solve(case, state):
    s = state["stepper"]
    s.upload_state(state["host"], 0.0, 0.0, 0.0, state["dts"])
    s.step(case["cycles"])
    s.download(state["out_np"])
    return {k: result(case, v) for k, v in state["out"].items()}


def run_history(case, state):
    s = state["stepper"]
    s.upload_state(state["host"], 0.0, 0.0, 0.0, state["dts"])
    frames = []
    for _ in range(case["frames"]):
        s.step(case["cycles"])
        s.download({"u": state["out_np"]["u"]})
        frames.append(result(case, state["out"]["u"]).clone())
    return frames


def run_output(case, state):
    s = state["stepper"]
    s.upload_state(state["host"], 0.0, 0.0, 0.0, state["dts"])
    s.step_until_async(case["cycles"], math.inf, math.inf)
    frames = []
    for k in range(case["frames"]):
        s.snapshot_begin()
        if k + 1 < case["frames"]:
            s.step_until_async(case["cycles"], math.inf, math.inf)
        sn = s.snapshot_wait()
        frames.append({f: result(case, sn[f]) for f in ("x", "u", "v", "a", "rf", "sigma")})
    s.sync()
    return frames


def run_sweep(case, state):
    b = state["batch"]
    slots = []
    for prep, p in zip(state["prepared"], state["problems"]):
        slot = b.add_prepared(prep)
        b.set_bcs(slot, p.bc_code, p.bc_value)
        b.arm(slot, case["cycles"])
        slots.append(slot)
    b.run(case["cycles"])
    b.sync()
    out = []
    for slot in slots:
        got = b.download(slot, ("u", "v", "sigma"))
        out.append(got)
        b.remove(slot)
    return {k: result(case, np.concatenate([o[k] for o in out])) for k in ("u", "v", "sigma")}


def run_serve(case, state):
    outcomes = S.Server(state["backend"], prepare_workers=4).serve(state["requests"])
    return {"u": result(case, np.concatenate([o.result["u"] for o in outcomes])),
            "cycles": np.array([o.cycles for o in outcomes]), "status": np.array([o.status for o in outcomes])}


# ---- what a pass cannot do without ------------------------------------------------

def sizes(case):
    """(elements, nodes, cycles) of each instance."""
    if case["kind"] in ("sweep", "serve"):
        return [(p.mesh.n_elements, p.mesh.n_nodes, p.cycles) for p in problems(case, 0)]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["shape"] == "bar":
        ne = (nx * nx + 4 * nx * ny) * nz
        nn = ((nx + 1) ** 2 + 4 * nx * ny) * (nz + 1)
    else:
        ne, nn = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    return [(ne, nn, case["cycles"] * case.get("frames", 1))]


def work(case):
    """Each cycle reads the mesh and the geometry of its elements (8 node numbers, the 3x3 matrix that gives the one-point
    B, V0) and the nodes (inverse mass, condition code), and reads and writes once the state the solve advances:
    sigma, hourglass history and plastic strain; x, u, v (mixed: x and v).  The hand-off of the element forces to
    the nodes is not counted.  Host state in, results out once.  The operations are those of the element update
    (about 900) and of the node update (about 50)."""
    mixed = case["precision"] == "mixed"
    elem = 32 + (72 + 8 + 4 + 2 * 19 * 4 if mixed else 72 + 24 + 2 * 19 * 8)
    node = 9 + (2 * (24 + 18) if mixed else 2 * 72)
    b = f = 0.0
    for ne, nn, cycles in sizes(case):
        b += cycles * (ne * elem + nn * node) + 8.0 * (19 * ne + 9 * nn) + 8.0 * (6 * ne + 6 * nn)
        f += cycles * (900.0 * ne + 50.0 * nn)
    return {"bytes": b, "flops": f}


# ---- 64-bit values ---------------------------------------------------------------

EDGES = ([0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3], [1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7])
CORNERS = [[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]]
GAMMA = [[1, -1, 1, -1, 1, -1, 1, -1], [-1, -1, 1, 1, 1, 1, -1, -1], [-1, 1, 1, -1, 1, -1, -1, 1],
         [-1, 1, -1, 1, 1, -1, 1, -1]]


class Solve64:
    """The explicit central-difference solve of several independent meshes in
    float64, plain torch: one-point hexahedra, Jaumann rate with J2 radial
    return, viscous and stiffness hourglass control, bulk viscosity."""

    def __init__(self, ps, device):
        dev, f64 = torch.device(device), torch.float64
        ten = lambda a, dt=f64: torch.as_tensor(np.asarray(a), device=dev).to(dt)  # noqa: E731
        off = np.cumsum([0] + [p.mesh.n_nodes for p in ps])
        self.conn = torch.cat([ten(p.mesh.conn.astype(np.int64), torch.int64) + int(o) for p, o in zip(ps, off)])
        self.ei = torch.cat([torch.full((p.mesh.n_elements,), i, device=dev) for i, p in enumerate(ps)])
        self.ni = torch.cat([torch.full((p.mesh.n_nodes,), i, device=dev) for i, p in enumerate(ps)])
        self.x = torch.cat([ten(p.mesh.x0) for p in ps])
        self.v = torch.cat([ten(p.v0) for p in ps])
        self.u = torch.zeros_like(self.x)
        code = torch.cat([ten(p.bc_code, torch.int64).reshape(-1, 3) for p in ps])
        value = torch.cat([ten(p.bc_value).reshape(-1, 3) for p in ps])
        self.fixed, self.driven, self.value = (code & 1) > 0, (code & 2) > 0, value
        self.n, self.ps = len(ps), ps
        per = lambda g: ten([g(p) for p in ps])  # noqa: E731
        E, nu = per(lambda p: p.material.E), per(lambda p: p.material.nu)
        self.rho = per(lambda p: p.material.rho)
        self.G = E / (2 * (1 + nu))
        self.K = E / (3 * (1 - 2 * nu))
        self.lam = 2 * self.G * nu / (1 - 2 * nu)
        self.c = torch.sqrt((self.lam + 2 * self.G) / self.rho)
        self.y0 = per(lambda p: p.material.yield_stress if p.material.yield_stress > 0 else math.inf)
        self.H = per(lambda p: p.material.hardening)
        for k in ("c_dr", "c_cr", "factor", "cvisl", "cvisq"):
            setattr(self, k, per(lambda p, k=k: getattr(p.controls, k)))
        ne = self.conn.shape[0]
        self.s = torch.zeros(ne, 6, dtype=f64, device=dev)
        self.q = torch.zeros(ne, 3, 4, dtype=f64, device=dev)
        self.ep = torch.zeros(ne, dtype=f64, device=dev)
        corner, self.gamma = ten(CORNERS), ten(GAMMA)
        jac = torch.einsum("jm,ejc->emc", corner / 8, self.x[self.conn])
        self.B = torch.einsum("ecm,jm->ejc", torch.linalg.inv(jac), corner / 8)  # (ne, 8, 3)
        self.V0 = 8 * torch.linalg.det(jac)
        self.bb = (self.B ** 2).sum((1, 2))
        m = (self.rho[self.ei] * self.V0 / 8)[:, None].expand(-1, 8)
        self.im = 1 / torch.zeros(len(self.x), dtype=f64, device=dev).index_add_(0, self.conn.reshape(-1),
                                                                                 m.reshape(-1))
        self.time = torch.zeros(self.n, dtype=f64, device=dev)
        self.dt = torch.zeros_like(self.time)
        self.a = self.rf = None
        self.dts = self.forces(torch.zeros_like(self.time), None)[2]
        self.v = torch.where(self.driven, self.value, self.v)
        self.v = torch.where(self.fixed, 0.0, self.v)

    def least(self, e):
        return torch.full((self.n,), math.inf, dtype=e.dtype, device=e.device).scatter_reduce_(0, self.ei, e, "amin")

    def forces(self, dt, live):
        ei = self.ei
        at = lambda p: p[ei]  # noqa: E731
        x, u, v = self.x[self.conn], self.u[self.conn], self.v[self.conn]
        edge = torch.sqrt(((x[:, EDGES[0]] - x[:, EDGES[1]]) ** 2).sum(-1).min(1).values)
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        F = eye + torch.einsum("eji,ejc->eic", u, self.B)
        J = torch.linalg.det(F)
        Fi = torch.linalg.inv(F)
        b = torch.einsum("ejc,ecd->ejd", self.B, Fi)
        L = torch.einsum("eji,ejc->eic", v, b)
        tau = self.gamma - torch.einsum("kj,ejc,eic->eki", self.gamma, x, self.B)  # (ne, 4, 8)
        vr = L.diagonal(dim1=1, dim2=2).sum(-1)
        h = at(dt)[:, None, None]
        D, Wm = (L + L.mT) / 2 * h, (L - L.mT) / 2 * h
        G, lam, V = at(self.G), at(self.lam), J * self.V0
        w0, w1, w2 = Wm[:, 0, 1], Wm[:, 0, 2], Wm[:, 1, 2]
        s0, s1, s2, s3, s4, s5 = self.s.unbind(1)
        # the solver's rotation terms (the shear rows as it has them)
        rate = torch.stack([2 * (s3 * w0 + s4 * w1), 2 * (s5 * w2 - s3 * w0), -2 * (s4 * w1 + s5 * w2),
                            (s1 - s0) * w0 + s5 * w1, (s2 - s0) * w1 + s5 * w0,
                            (s2 - s1) * w2 + s3 * w1 - s4 * w0], 1)
        new = self.full(self.s + rate) + 2 * G[:, None, None] * D \
            + (lam * D.diagonal(dim1=1, dim2=2).sum(-1))[:, None, None] * eye
        pm = new.diagonal(dim1=1, dim2=2).sum(-1)[:, None, None] / 3 * eye
        dev = new - pm
        seq = torch.sqrt(1.5 * (dev ** 2).sum((1, 2)))
        over = seq - (at(self.y0) + at(self.H) * self.ep)
        yields = over > 0
        dl = torch.where(yields, over / (3 * G + at(self.H)), 0.0)
        r = torch.where(yields, 1 - 3 * G * dl / torch.where(yields, seq, 1.0), 1.0)
        new = pm + dev * r[:, None, None]
        hia = torch.einsum("eji,ekj->eik", v, tau)
        DR = at(self.c_dr) * (4 / 3 * G + at(self.K)) * 0.1 * self.bb * V / math.sqrt(8.0) * at(dt)
        CR = at(self.c_cr) * at(self.rho) / J * (self.V0 ** 2) ** (1 / 3) * at(self.c) / 4
        q = self.q + DR[:, None, None] * hia
        l0 = self.V0 ** (1 / 3)
        m0 = vr.clamp(max=0.0)
        pv = at(self.rho) / J * l0 * (at(self.cvisq) ** 2 * l0 * vr * m0 - at(self.cvisl) * at(self.c) * vr)
        pv = torch.where(vr.abs() < 1e-10, 0.0, pv)
        f = -V[:, None, None] * torch.einsum("ejc,ecd->ejd", b, new - pv[:, None, None] * eye) \
            - torch.einsum("ekj,eik->eji", tau, q + CR[:, None, None] * hia)
        xi = at(self.cvisl) - at(self.cvisq) ** 2 * edge / at(self.c) * m0
        dts = (torch.sqrt(1 + xi * xi) - xi) * edge / at(self.c)
        if live is not None:
            on = live[ei]
            flat = torch.stack([new[:, 0, 0], new[:, 1, 1], new[:, 2, 2], new[:, 0, 1], new[:, 0, 2], new[:, 1, 2]], 1)
            self.s = torch.where(on[:, None], flat, self.s)
            self.q = torch.where(on[:, None, None], q, self.q)
            self.ep = torch.where(on, self.ep + dl, self.ep)
        total = torch.zeros_like(self.x).index_add_(0, self.conn.reshape(-1), f.reshape(-1, 3))
        return total, self.least(edge), self.least(dts)

    @staticmethod
    def full(s):
        return torch.stack([s[:, 0], s[:, 3], s[:, 4], s[:, 3], s[:, 1], s[:, 5], s[:, 4], s[:, 5], s[:, 2]],
                           1).reshape(-1, 3, 3)

    def cycle(self, live):
        dt1 = self.dt
        self.time = torch.where(live, self.time + dt1, self.time)
        f, edge, dts = self.forces(dt1, live)
        dt = torch.minimum(edge / self.c, self.dts) * self.factor
        for i, p in enumerate(self.ps):
            if p.controls.gravity is not None:
                value, direction = p.controls.gravity
                g = value * torch.tensor(direction, dtype=f.dtype, device=f.device)
                amp = amplitude(p.controls.gravity_amplitude, float(self.time[i]), float(dt[i]))
                f = f + torch.where((self.ni == i)[:, None], amp * g / self.im[:, None], 0.0)
        self.rf = torch.where(self.fixed & ~self.driven, -f, 0.0)
        f = torch.where(self.fixed | self.driven, 0.0, f)
        self.a = f * self.im[:, None]
        on = live[self.ni][:, None]
        self.v = torch.where(on, self.v + ((dt + dt1) / 2)[self.ni][:, None] * self.a, self.v)
        step = torch.where(on, dt[self.ni][:, None] * self.v, 0.0)
        self.u = self.u + step
        self.x = self.x + step
        self.dt = torch.where(live, dt, self.dt)
        self.dts = torch.where(live, dts, self.dts)

    def run(self, cycles):
        cycles = torch.as_tensor(cycles, device=self.x.device)
        for k in range(int(cycles.max())):
            self.cycle(cycles > k)


def amplitude(points, time, dt):
    """The amplitude factor of a cycle from `time` to `time + dt`: the curve at mid-cycle, and for a cycle over a
    point of the table the mean over its parts, the last of them with the first segment's slope in its
    intercept."""
    if not points or len(points) < 2:
        return 1.0
    for i in range(len(points) - 1):
        (x1, y1), (x2, y2) = points[i], points[i + 1]
        if time > x2:
            return 1.0
        m = (y2 - y1) / (x2 - x1)
        if time + dt < x2:
            return y1 + m * (time + dt / 2 - x1)
        total = (y1 + m * (time + (x2 - time) / 2 - x1)) * (x2 - time)
        for j in range(i + 2, len(points)):
            (xp, yp), (xj, yj) = points[j - 1], points[j]
            if time + dt > xj:
                total += (xj - xp) * (yj + yp) / 2
            else:
                end = (yj - yp) / (xj - xp) * (time + dt) + (yp - m * xp)
                total += (time + dt - xp) * (yp + end) / 2
                break
        if time + dt > points[-1][0]:
            total += time + dt - points[-1][0]
        return total / dt
    return 1.0


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] in ("sweep", "serve"):
        ps = problems(case, seed)
        w = Solve64(ps, device)
        w.run([p.cycles for p in ps])
        if case["kind"] == "serve":
            return {"u": w.u, "cycles": None, "status": None}
        return {"u": w.u, "v": w.v, "sigma": w.s}
    w = Solve64([problem(case, seed)], device)
    if case["kind"] == "solve":
        w.run([case["cycles"]])
        got = {"u": w.u, "v": w.v, "sigma": w.s}
        return {**got, "x": w.x, "qia": w.q.reshape(-1, 12), "eps_p": w.ep} if case["checkpoint"] else got
    frames = []
    for _ in range(case["frames"]):
        w.run([case["cycles"]])
        if case["kind"] == "history":
            frames.append(w.u)
        else:
            frames.append({"x": w.x, "u": w.u, "v": w.v, "a": w.a, "rf": w.rf, "sigma": w.s})
    return frames
