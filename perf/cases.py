"""The work that a coupled LB-DEM program has this framework do, as timed cases.

Every case goes through the Python face of the C ABI (``lbdem.Lattice`` and
``lbdem.Batch``) the way a coupling program calls it.  Kinds:

* ``cycle``    one coupling cycle with host buffers: this step's particle list in,
               voxelization, collide-stream, forces and torques out (what a host
               DEM does in every lattice step);
* ``device``   the same cycle with the particle table and the force sums in device
               memory and no synchronisation (a DEM that lives on the GPU);
* ``batch``    one coupling cycle of many independent channels of uneven size;
* ``adjoint``  one window of steps with its gradients (parameter fitting);
* ``restart``  populations in, a few cycles, the populations and the exported fields out
               (checkpoints, and what is written every some hundred steps).

Spheres sit on a jittered grid (no overlaps) and shuttle with their velocities
around their places, so that a case can be run any number of times: the
prescribed motion stays in the range in which the scheme is stable.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "lbdemcoupling-public_gb300"))
import lbdem  # noqa: E402

FP64, FP32 = "fp64", "fp32"
HALF = 6           # steps that the spheres move one way before they turn
PHASES = 2 * HALF
GRAVITY = 1e-6     # body force, lattice units


def listed():
    return [
        # The smallest call: a tiny periodic box in the drop-in form, with the default tag
        # range of a handle, where launches and latency are all there is.
        _cycle("cycle_box_24x20x28_fp64", (24, 20, 28), "ppp", FP64, 4, 3.0, 3.5, tau=0.6, max_tag=1 << 20),
        # The reference's plain case: one sphere settling in a closed 60x60x180 box.
        _cycle("cycle_settling_60x60x180_fp64", (60, 60, 180), "www", FP64, 1, 5.0, 5.0, tau=0.6, max_tag=16),
        # An ordinary suspension in the drop-in form.
        _cycle("cycle_suspension_128_fp64", (128, 128, 128), "ppp", FP64, 250, 8.0, 8.0, tau=0.55),
        # The headline workload: periodic 256^3, about 2000 spheres r = 8, the fast form.
        _cycle("cycle_suspension_256_fp32", (256, 256, 256), "ppp", FP32, 2000, 8.0, 8.0, tau=0.55),
        # The largest: a packed polydisperse bed with the flow driven by a body force.
        _cycle("cycle_bed_512x256x256_fp32", (512, 256, 256), "ppp", FP32, 8000, 5.0, 7.0, tau=0.6, force=True,
               vel=0.0),
        # A pressure-driven channel with odd extents (rows that are not 16-byte aligned).
        _cycle("cycle_channel_71x67x243_fp32", (71, 67, 243), "wwp", FP32, 60, 4.0, 6.0, tau=0.6, drop=2),
        # The same kind of channel in the drop-in form, flow along x as in the showcase.
        _cycle("cycle_channel_160x48x50_fp64", (160, 48, 50), "pww", FP64, 30, 4.0, 5.0, tau=0.6, drop=0),
        # A GPU-resident DEM on an ordinary suspension.
        dict(_cycle("device_suspension_96_fp32", (96, 96, 96), "ppp", FP32, 110, 8.0, 8.0, tau=0.55), kind="device"),
        # Parameter sweeps: many uneven pressure-driven channels in one batch.
        {"name": "batch_512_channels_fp32", "kind": "batch", "prec": FP32, "domains": 512, "lmin": 64, "lmax": 160,
         "wmin": 24, "wmax": 48, "tau": 0.6},
        # Gradients over a window of steps: the fast form and the drop-in form.
        {"name": "adjoint_128_fp32", "kind": "adjoint", "prec": FP32, "nx": 128, "ny": 128, "nz": 128, "n": 64,
         "r": 6.0, "tau": 0.6, "steps": 20, "every": 10, "want_f0": False},
        {"name": "adjoint_64_fp64", "kind": "adjoint", "prec": FP64, "nx": 64, "ny": 64, "nz": 64, "n": 27,
         "r": 6.0, "tau": 0.6, "steps": 12, "every": 4, "want_f0": True},
        # Restart and output: the whole state in, five cycles, the state and the fields out.
        dict(_cycle("restart_72x64x80_fp64", (72, 64, 80), "ppp", FP64, 27, 6.0, 7.0, tau=0.6), kind="restart",
             cycles=5),
    ]


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["cycle"] * 5 + ["device", "batch", "adjoint", "restart"])
    prec = rng.choice([FP64, FP32])
    tau = rng.choice([0.55, 0.6, 0.8])

    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "batch":
        wmin, lmin = rng.randint(16, 32), rng.randint(33, 96)
        return {"kind": kind, "prec": prec, "domains": side(4, 400 if prec == FP32 else 64), "lmin": lmin,
                "lmax": lmin + rng.randint(0, 64), "wmin": wmin, "wmax": wmin + rng.randint(0, 16), "tau": tau}
    if kind == "adjoint":
        hi = 120 if prec == FP32 else 80
        s = [side(30, hi) for _ in range(3)]
        r = rng.uniform(4.0, 6.5)
        steps = rng.randint(3, 16)
        return {"kind": kind, "prec": prec, "nx": s[0], "ny": s[1], "nz": s[2], "r": r, "tau": tau, "steps": steps,
                "n": _fit(s, r, rng.uniform(0.2, 0.8)), "every": rng.randint(1, steps), "want_f0": rng.random() < 0.3}
    hi = 96 if kind == "restart" else 256
    s = [side(20, hi) for _ in range(3)]
    rmin = rng.uniform(2.5, 7.0)
    rmax = min(rmin * rng.uniform(1.0, 1.6), (min(s) - 8) / 2)
    rmin = min(rmin, rmax)
    form = rng.choice(["plain", "plain", "force", "drop"])
    per, drop = rng.choice(["ppp", "ppp", "www", "pww", "wwp", "ppw"]), None
    if form == "drop":
        drop = rng.choice([0, 2])
        per = "pww" if drop == 0 else "wwp"
    c = _cycle("", s, per, prec, _fit(s, rmax, rng.uniform(0.1, 1.0)), rmin, rmax, tau=tau, force=form == "force",
               drop=drop, max_tag=rng.choice([0, 0, 4000, 1 << 20]))
    c["kind"] = kind
    if kind == "restart":
        c["cycles"] = rng.randint(2, 6)
    del c["name"]
    return c


def _cycle(name, shape, per, prec, n, rmin, rmax, tau, force=False, drop=None, max_tag=0, vel=0.002):
    return {"name": name, "kind": "cycle", "nx": shape[0], "ny": shape[1], "nz": shape[2], "per": per, "prec": prec,
            "n": n, "rmin": rmin, "rmax": rmax, "tau": tau, "force": force, "drop": drop, "max_tag": max_tag,
            "vel": vel}


def _slots(shape, r):
    """Places of a jittered grid along each axis for spheres up to radius r."""
    return [max(1, int((s - 6) // (2.0 * r + 1.2))) for s in shape]


def _fit(shape, r, share):
    return max(1, int(share * np.prod(_slots(shape, r))))


# ---- inputs ------------------------------------------------------------------

def _rng(seed, salt=0):
    return np.random.default_rng([int(seed) & 0xffffffff, salt])


def _place(rng, shape, per, n, rmin, rmax, vel):
    """n spheres on a jittered grid, at rest (vel 0) or with velocities N(0, vel)."""
    k = _slots(shape, rmax)
    n = min(n, int(np.prod(k)))
    at = np.stack(np.unravel_index(rng.permutation(int(np.prod(k)))[:n], k), axis=1)
    L = np.array(shape, dtype=np.float64)
    pad = np.array([0.0 if p == "p" else 3.0 for p in per])
    pitch = (L - 2 * pad) / np.array(k)
    r = rng.uniform(rmin, rmax, n)
    free = np.maximum(0.0, pitch[None, :] / 2 - r[:, None] - 0.15)
    x = pad + (at + 0.5) * pitch + rng.uniform(-1, 1, (n, 3)) * free
    v = np.clip(rng.normal(0.0, 1.0, (n, 3)), -3, 3) * vel
    w = np.clip(rng.normal(0.0, 1.0, (n, 3)), -3, 3) * vel / 10
    return x, v, w, r


def _with_images(x, v, w, r, tag, shape, per):
    """The list a DEM hands over: owned spheres, then their periodic images that reach the lattice."""
    for a in range(3):
        if per[a] != "p":
            continue
        up = np.nonzero(x[:, a] - r - 2.0 < 0.0)[0]
        dn = np.nonzero(x[:, a] + r + 2.0 > shape[a] - 1.0)[0]
        idx = np.concatenate([up, dn])
        xi = x[idx].copy()
        xi[:, a] += np.concatenate([np.full(up.size, float(shape[a])), np.full(dn.size, -float(shape[a]))])
        x, v, w = np.concatenate([x, xi]), np.concatenate([v, v[idx]]), np.concatenate([w, w[idx]])
        r, tag = np.concatenate([r, r[idx]]), np.concatenate([tag, tag[idx]])
    return tuple(np.ascontiguousarray(b) for b in (x, v, w, r)) + (np.ascontiguousarray(tag, dtype=np.int32),)


def _lists(x, v, w, r, shape, per):
    """The particle lists of the PHASES steps of the spheres' shuttling motion."""
    tag = np.arange(1, x.shape[0] + 1, dtype=np.int32)
    L = np.array(shape, dtype=np.float64)
    out = []
    for t in range(PHASES):
        sign = 1.0 if t < HALF else -1.0
        q = x + (t if t <= HALF else PHASES - t) * v
        for a in range(3):
            if per[a] == "p":
                q[:, a] = np.mod(q[:, a], L[a])
        out.append(_with_images(q, sign * v, sign * w, r, tag, shape, per))
    return out


def _records(p):
    x, v, w, r, tag = p
    rec = np.zeros((x.shape[0], 12))
    rec[:, 0:3], rec[:, 3:6], rec[:, 6:9], rec[:, 9], rec[:, 10] = x, v, w, r, tag
    return rec


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _scene(case, seed):
    shape = _shape(case)
    return _lists(*_place(_rng(seed), shape, case["per"], case["n"], case["rmin"], case["rmax"], case["vel"]), shape,
                  case["per"])


def _drop_of(shape, axis):
    """Inlet and outlet boxes (first and last plane, interior rows) of a pressure-driven channel."""
    box = [1, shape[0] - 2, 1, shape[1] - 2, 1, shape[2] - 2]
    inlet, outlet = list(box), list(box)
    inlet[2 * axis] = inlet[2 * axis + 1] = 0
    outlet[2 * axis] = outlet[2 * axis + 1] = shape[axis] - 1
    return inlet, outlet


def _room(case):
    """Rows of a DEM's arrays: the owned spheres and every image they can have."""
    return min(case["n"], int(np.prod(_slots(_shape(case), case["rmax"])))) * 2 ** case["per"].count("p")


def _rows(a, rows, axis=0):
    """a in an array with room for `rows` entries along an axis."""
    full = list(a.shape)
    full[axis] = rows
    out = torch.zeros(full, dtype=a.dtype) if torch.is_tensor(a) else np.zeros(full)
    out[(slice(None),) * axis + (slice(0, a.shape[axis]),)] = a
    return out


RHO_IN, RHO_OUT, U_MAX, U_0 = 1.0, 0.999, 0.01, 0.01


def _prec(case):
    return lbdem.PREC_FP64 if case["prec"] == FP64 else lbdem.PREC_FP32_DEV


def _lattice(case, lists):
    shape = _shape(case)
    most = max(p[3].size for p in lists)
    top = int(max(p[4].max() for p in lists))
    lat = lbdem.Lattice(*shape, 1.0 / case["tau"], periodic=[int(c == "p") for c in case["per"]],
                        precision=_prec(case), body_force=(GRAVITY if case["force"] else 0.0, 0.0, 0.0),
                        max_particles=most, max_tag=max(case["max_tag"], top), max_radius=16.0)
    if case["drop"] is not None:
        inlet, outlet = _drop_of(shape, case["drop"])
        lat.set_pressure_drop(case["drop"], inlet, outlet, rho_in=RHO_IN, rho_out=RHO_OUT)
        lat.init_profile(1, RHO_IN, RHO_OUT, U_MAX, shape, case["drop"])
    elif case["per"] == "ppp":
        lat.init_equilibrium(0.0, (U_0, 0.0, 0.0))
    return lat


def _warm(case):
    """Cycles before the timed one, so that the flow around the spheres has begun."""
    return 6 if case["nx"] * case["ny"] * case["nz"] < 4_000_000 else 2


def _populations(case, seed):
    """Populations of a smooth random flow with some non-equilibrium part, [19][nx][ny][nz]."""
    rng = _rng(seed, 1)
    X = np.meshgrid(*[2 * np.pi * np.arange(s) / s for s in _shape(case)], indexing="ij")
    j = np.stack([sum(0.01 * rng.normal() * np.sin(X[a] + 2 * np.pi * rng.random()) for a in range(3))
                  for _ in range(3)])
    rb = sum(1e-3 * rng.normal() * np.cos(X[a]) for a in range(3))
    f = np.empty((19,) + _shape(case))
    for i in range(19):
        cj = C[i][0] * j[0] + C[i][1] * j[1] + C[i][2] * j[2]
        f[i] = W[i] * (rb + 3 * cj + 4.5 * cj * cj - 1.5 * (j * j).sum(0))
    f += 1e-5 * rng.standard_normal(f.shape)
    return f.astype(np.float64 if case["prec"] == FP64 else np.float32)


def _domains(case, seed):
    sizes, rng = _rng(case["domains"], case["lmax"]), _rng(seed)
    doms, lists = [], []
    for _ in range(case["domains"]):
        length, width = int(sizes.integers(case["lmin"], case["lmax"] + 1)), int(sizes.integers(case["wmin"], case["wmax"] + 1))
        shape = (width, width, length)
        inlet, outlet = _drop_of(shape, 2)
        scene = _lists(*_place(rng, shape, "wwp", int(sizes.integers(1, 41)), 3.0, min(6.0, (width - 8) / 2.0), 0.002),
                       shape, "wwp")
        doms.append({"shape": shape, "periodic": (0, 0, 1), "omega": 1.0 / case["tau"],
                     "max_particles": max(p[3].size for p in scene),
                     "drop": {"dimension": 2, "inlet": inlet, "outlet": outlet, "rho_in": RHO_IN, "rho_out": RHO_OUT}})
        lists.append(scene)
    steps = []
    for t in range(PHASES):
        steps.append((np.array([s[t][3].size for s in lists], dtype=np.int32),
                      np.concatenate([_records(s[t]) for s in lists]), [{"n": int(s[t][4].max())} for s in lists]))
    return doms, steps


def _window_room(case):
    return 8 * min(case["n"], int(np.prod(_slots(_shape(case), case["r"]))))


def _window(case, seed):
    shape, steps = _shape(case), case["steps"]
    x, v, w, r = _place(_rng(seed), shape, "ppp", case["n"], case["r"], case["r"], 0.002)
    tag = np.arange(1, x.shape[0] + 1, dtype=np.int32)
    p = _with_images(x, v, w, r, tag, shape, "ppp")
    rec = np.repeat(_records(p)[None], steps, axis=0)
    # velocities that change from step to step, as in a fit of a prescribed motion
    wave = 1.0 + 0.1 * np.sin(0.7 * np.arange(steps))[:, None, None]
    rec[:, :, 3:9] *= wave
    rng = _rng(seed, 2)
    weights = np.zeros((steps, rec.shape[1], 6))
    weights[:, :x.shape[0], :3] = rng.normal(1.0, 0.3, (steps, x.shape[0], 3))
    weights[:, :x.shape[0], 3:] = rng.normal(0.0, 0.05, (steps, x.shape[0], 3))
    return rec, weights


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "t": 0, "case": case}
    if kind == "batch":
        doms, steps = _domains(case, seed)
        b = lbdem.Batch(doms, precision=_prec(case), max_tag=64, max_radius=8.0)
        for d, dom in enumerate(doms):
            b.init_profile(d, 1, RHO_IN, RHO_OUT, U_MAX, dom["shape"], 2)
        room = 2 * int(sum(s["n"] for s in steps[0][2]))
        state.update(batch=b, steps=[s[:2] for s in steps], F=np.zeros((room, 3)), T=np.zeros((room, 3)))
        for _ in range(4):   # the first steps tune and capture
            run(state)
        return state
    if kind == "adjoint":
        rec, weights = _window(case, seed)
        lat = lbdem.Lattice(*_shape(case), 1.0 / case["tau"], precision=_prec(case), body_force=(GRAVITY, 0.0, 0.0),
                            max_particles=rec.shape[1], max_tag=rec.shape[1] + 1, max_radius=8.0)
        lat.init_equilibrium(0.0, (U_0, 0.0, 0.0))
        state.update(lat=lat, rec=rec, weights=weights, room=_window_room(case))
        return state
    lists = _scene(case, seed)
    lat = _lattice(case, lists)
    state.update(lat=lat, lists=lists, F=np.zeros((_room(case), 3)), T=np.zeros((_room(case), 3)))
    if kind == "restart":
        state["f"] = _populations(case, seed)
        return state
    for _ in range(_warm(case)):
        lat.cycle(*lists[state["t"] % PHASES])
        state["t"] += 1
    if kind == "device":
        state["rec"] = [torch.from_numpy(_records(p)).cuda() for p in lists]
        state["ft"] = torch.zeros(6 * _room(case), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
    return state


def run(state):
    kind, t = state["kind"], state["t"] % PHASES
    if kind == "batch":
        state["t"] += 1
        force, torque = state["batch"].cycle(*state["steps"][t])
        state["F"][:force.shape[0]] = force
        state["T"][:torque.shape[0]] = torque
        return state["F"], state["T"]
    lat = state["lat"]
    if kind == "cycle":
        state["t"] += 1
        return lat.cycle(*state["lists"][t], F=state["F"], T=state["T"])
    if kind == "device":
        state["t"] += 1
        rec, ft = state["rec"][t], state["ft"]
        lat.set_particles_device(rec.shape[0], rec.data_ptr())
        lat.collide_and_stream()
        lat.get_forces_device(ft.data_ptr())
        return ft
    if kind == "adjoint":
        out = lat.adjoint_window(state["rec"], state["weights"], state["case"]["every"], state["case"]["want_f0"])
        out["grad_vel"] = _rows(out["grad_vel"], state["room"], 1)
        return out
    lat.set_populations(state["f"])   # restart
    for k in range(state["case"]["cycles"]):
        force, torque = lat.cycle(*state["lists"][k], F=state["F"], T=state["T"])
    return {"force": force, "torque": torque, "populations": lat.get_populations(),
            "density": lat.get_field(lbdem.FIELD_DENSITY), "velocity": lat.get_field(lbdem.FIELD_VELOCITY)}


def work(case):
    kind = case["kind"]
    size = 8 if case["prec"] == FP64 else 4
    step = 2 * 19 * size + 4     # a cell's populations read and written, its voxel word
    flops = 250                  # a cell's collision
    if kind == "batch":
        cells = case["domains"] * (case["wmin"] + case["wmax"]) ** 2 / 4 * (case["lmin"] + case["lmax"]) / 2
        return {"bytes": step * cells, "flops": flops * cells}
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "adjoint":
        # every step forward once; in reverse the populations and the incoming and outgoing adjoint
        return {"bytes": case["steps"] * cells * (step + 3 * 19 * size + 4), "flops": case["steps"] * cells * 900}
    if kind == "restart":
        return {"bytes": cells * (case["cycles"] * step + 2 * 19 * size + 4 * 8), "flops": case["cycles"] * flops * cells}
    return {"bytes": step * cells, "flops": flops * cells}


# ---- the same in 64 bits, in plain torch ---------------------------------------

C = [(0, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (-1, -1, 0), (-1, 1, 0), (-1, 0, -1), (-1, 0, 1), (0, -1, -1),
     (0, -1, 1)]
C = C + [(-a, -b, -c) for a, b, c in C[1:]]
W = [1 / 3] + [1 / 18 if sum(abs(q) for q in c) == 1 else 1 / 36 for c in C[1:]]
DELTA = [-0.5 + (i + 0.5) * (1.0 / 5.0) for i in range(5)]


def _opp(i):
    return 0 if i == 0 else (i + 9 if i <= 9 else i - 9)


class _Exact:
    """The coupled lattice in float64: a cell's populations f - t, its solid count, owner and surface velocity."""

    def __init__(self, shape, per, tau, force):
        self.shape, self.per, self.omega = shape, [c == "p" for c in per], 1.0 / tau
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        kw = {"dtype": torch.float64, "device": self.dev}
        self.f = torch.zeros((19,) + tuple(shape), **kw)
        self.n = torch.zeros(tuple(shape), **kw)
        self.id = torch.zeros(tuple(shape), dtype=torch.int64, device=self.dev)
        self.up = torch.zeros((3,) + tuple(shape), **kw)
        self.g = [GRAVITY if force else 0.0, 0.0, 0.0]
        self.kw = kw
        self.beyond = []
        for c in C:
            m = torch.zeros(tuple(shape), dtype=torch.bool, device=self.dev)
            for a in range(3):
                if c[a] != 0 and not self.per[a]:
                    m.select(a, 0 if c[a] > 0 else shape[a] - 1).fill_(True)
            self.beyond.append(m if bool(m.any()) else None)

    def equilibrium(self, rho_bar, u):
        """rho_bar, u[3]: numbers or fields."""
        rb = rho_bar if torch.is_tensor(rho_bar) else torch.full(tuple(self.shape), rho_bar, **self.kw)
        j = [(1 + rb) * q for q in u]
        for i in range(19):
            self.f[i] = _feq(i, rb, j, 1 / (1 + rb))

    def profile(self, axis):
        at = [torch.arange(s, **self.kw).reshape([-1 if a == d else 1 for d in range(3)])
              for a, s in enumerate(self.shape)]
        rho = RHO_IN - (RHO_IN - RHO_OUT) * at[axis] / (self.shape[axis] - 1)
        u = [torch.zeros(tuple(self.shape), **self.kw) for _ in range(3)]
        across = [a for a in range(3) if a != axis]
        half = [self.shape[a] / 2.0 for a in across]
        shape_of = [1 - ((at[a] - h) / h) ** 2 for a, h in zip(across, half)]
        u[axis] = U_MAX * shape_of[0] * shape_of[1] + u[axis]
        self.equilibrium((rho - 1) + torch.zeros(tuple(self.shape), **self.kw), u)

    def spheres(self, x, v, w, r, tag):
        """Every sphere in list order: solid counts, owners and surface velocities."""
        s31 = math.sqrt(3.1) / 2
        dl = torch.tensor(DELTA, **self.kw)
        self.first = {}
        for k in range(x.shape[0]):
            self.first.setdefault(int(tag[k]), k)
            lo = [max(0, int(x[k, a] - r[k] - 2.0)) for a in range(3)]
            hi = [min(self.shape[a] - 1, int(x[k, a] + r[k] + 2.0)) for a in range(3)]
            if any(l > h for l, h in zip(lo, hi)):
                continue
            box = tuple(slice(l, h + 1) for l, h in zip(lo, hi))
            d = [(torch.arange(lo[a], hi[a] + 1, **self.kw) - float(x[k, a])).reshape([-1 if a == b else 1 for b in range(3)])
                 for a in range(3)]
            dist = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
            rp, rm, rsq = float(r[k]) + s31, float(r[k]) - s31, float(r[k]) * float(r[k])
            n = 125.0 * (dist < rm * rm).to(torch.float64)
            shell = torch.nonzero(~(dist > rp * rp) & ~(dist < rm * rm), as_tuple=True)
            s = [(d[a].reshape(-1)[shell[a]][:, None] + dl) ** 2 for a in range(3)]
            t = (s[0][:, :, None, None] + s[1][:, None, :, None]) + s[2][:, None, None, :]
            n[shell] = (t < rsq).to(torch.float64).sum((1, 2, 3))
            old, own = self.n[box], self.id[box]
            mine = own == int(tag[k])
            clear = (n == 0) & (old > 0) & mine
            put = (n > 0) & ((old == 0) | (n > old) | mine)
            self.n[box] = torch.where(put, n, torch.where(clear, torch.zeros_like(n), old))
            self.id[box] = torch.where(put, torch.full_like(own, int(tag[k])), torch.where(clear, torch.zeros_like(own), own))
            u = [v[k, 0] + (w[k, 1] * d[2] - w[k, 2] * d[1]), v[k, 1] + (-w[k, 0] * d[2] + w[k, 2] * d[0]),
                 v[k, 2] + (w[k, 0] * d[1] - w[k, 1] * d[0])]
            for a in range(3):
                now = self.up[a][box]
                self.up[a][box] = torch.where(put, u[a] + torch.zeros_like(n), torch.where(clear, torch.zeros_like(n), now))
        self.x = x

    def owners(self):
        slot = torch.full((int(max(self.first)) + 1,), -1, dtype=torch.int64, device=self.dev)
        for t, k in self.first.items():
            slot[t] = k
        return torch.where(self.n > 0, slot[torch.where(self.n > 0, self.id, torch.zeros_like(self.id))],
                           torch.full_like(self.id, -1))

    def arms(self, owner):
        xs = torch.tensor(self.x, **self.kw)[owner.clamp(min=0)]
        out = []
        for a in range(3):
            L, h = self.shape[a], self.shape[a] // 2
            d = torch.arange(L, **self.kw).reshape([-1 if a == b else 1 for b in range(3)]) - xs[..., a]
            out.append(torch.where(d > h, d - L, torch.where(d < -h, d + L, d)))
        return out

    def collide(self, f, up, omega, g):
        """Post-collision populations and the force on every cell's particle."""
        rb = f.sum(0)
        j = _momentum(f)
        rho, r = 1 + rb, 1 / (1 + rb)
        J = [j[a] + 0.5 * rho * g[a] for a in range(3)]
        u = [q * r for q in J]
        ug = u[0] * g[0] + u[1] * g[1] + u[2] * g[2]
        pre = (1 - 0.5 * omega) * rho
        full = self.n == 125
        fs = []
        for i in range(19):
            cu, cg = _dot(i, u), _dot(i, g)
            src = W[i] * pre * (3 * (cg - ug) + 9 * cu * cg)
            fs.append(torch.where(full, f[i], (1 - omega) * f[i] + omega * _feq(i, rb, J, r) + src))
        fs = torch.stack(fs)
        rbs, js = fs.sum(0), _momentum(fs)
        rs = 1 / (1 + rbs)
        P = [(1 + rbs) * up[a] for a in range(3)]
        ooo = 1.0 / omega - 0.5
        sf = self.n / 125.0
        B = torch.where(full, torch.ones_like(sf), sf * ooo / ((1 - sf) + ooo))
        out = []
        for i in range(19):
            o = _opp(i)
            if i == 0:
                bb = f[0] + _feq(0, rbs, js, rs) - _feq(0, rbs, P, rs)
            else:
                bb = f[o] - _feq(o, rbs, js, rs) + _feq(i, rbs, P, rs)
            out.append(torch.where(self.n > 0, (1 - B) * fs[i] + B * bb, fs[i]))
        F = [torch.where(self.n > 0, B * (2 * j[a] - js[a] - P[a]), torch.zeros_like(B)) for a in range(3)]
        return torch.stack(out), F

    def stream(self, out):
        new = []
        for i in range(19):
            m = torch.roll(out[i], shifts=C[i], dims=(0, 1, 2))
            new.append(m if self.beyond[i] is None else torch.where(self.beyond[i], out[_opp(i)], m))
        return torch.stack(new)

    def sums(self, F, owner, arm, n):
        """Force and torque of every list entry."""
        at = owner.reshape(-1).clamp(min=0)
        T = [arm[1] * F[2] - arm[2] * F[1], arm[2] * F[0] - arm[0] * F[2], arm[0] * F[1] - arm[1] * F[0]]
        both = []
        for q in (F, T):
            both.append(torch.stack([torch.zeros(n, **self.kw).index_add(0, at, torch.where(
                owner >= 0, c, torch.zeros_like(c)).reshape(-1)) for c in q], dim=1))
        return both

    def step(self, p, drop):
        self.spheres(*p)
        if drop is not None:
            boxes = [tuple(slice(b[2 * a], b[2 * a + 1] + 1) for a in range(3)) for b in _drop_of(self.shape, drop)]
            mean = [1 + float(self.f.sum(0)[b].mean()) for b in boxes]
        out, F = self.collide(self.f, self.up, self.omega, self.g)
        owner = self.owners()
        both = self.sums(F, owner, self.arms(owner), p[3].size)
        self.f = self.stream(out)
        if drop is not None:
            for b, way, ratio in ((boxes[0], 1, RHO_IN / mean[1]), (boxes[1], -1, RHO_OUT / mean[0])):
                for i in range(19):
                    if C[i][drop] == way:
                        self.f[i][b] = (self.f[i][b] + W[i]) * ratio - W[i]
        return both


def _dot(i, q):
    s = 0.0
    for a in range(3):
        if C[i][a]:
            s = s + C[i][a] * q[a]
    return s


def _momentum(f):
    return [sum(C[i][a] * f[i] for i in range(19) if C[i][a]) for a in range(3)]


def _feq(i, rb, j, r):
    cj = _dot(i, j)
    return W[i] * (rb + 3 * cj + r * (4.5 * cj * cj - 1.5 * (j[0] * j[0] + j[1] * j[1] + j[2] * j[2])))


def _start(case):
    e = _Exact(_shape(case), case["per"], case["tau"], case["force"])
    if case["drop"] is not None:
        e.profile(case["drop"])
    elif case["per"] == "ppp":
        e.equilibrium(0.0, (U_0, 0.0, 0.0))
    return e


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "adjoint":
        return _exact_window(case, seed) if cells * case["steps"] <= 3_500_000 else None
    if cells > 2_200_000 or case["n"] > 700:
        return None
    lists, room = _scene(case, seed), _room(case)
    e = _start(case)
    if kind == "restart":
        e.f = torch.tensor(_populations(case, seed), **e.kw)
        for k in range(case["cycles"]):
            both = e.step(lists[k], case["drop"])
        rho = 1 + e.f.sum(0)
        return {"force": _rows(both[0].cpu(), room), "torque": _rows(both[1].cpu(), room), "populations": e.f.cpu(), "density": rho.cpu(),
                "velocity": torch.stack([q / rho for q in _momentum(e.f)]).cpu()}
    for k in range(_warm(case)):
        e.step(lists[k % PHASES], case["drop"])
    F, T = e.step(lists[_warm(case) % PHASES], case["drop"])
    if kind == "device":
        return _rows(torch.cat([F.reshape(-1), T.reshape(-1)]).cpu(), 6 * room)
    return _rows(F.cpu(), room), _rows(T.cpu(), room)


def _exact_window(case, seed):
    """The window's loss and gradients by automatic differentiation."""
    rec, weights = _window(case, seed)
    e = _Exact(_shape(case), "ppp", case["tau"], True)
    e.equilibrium(0.0, (U_0, 0.0, 0.0))
    n = rec.shape[1]
    e.spheres(rec[0, :, 0:3], rec[0, :, 3:6], rec[0, :, 6:9], rec[0, :, 9], rec[0, :, 10].astype(np.int64))
    owner = e.owners()
    solid, at = owner >= 0, owner.clamp(min=0)
    d = e.arms(owner)
    vel = torch.tensor(rec[:, :, 3:9], requires_grad=True, **e.kw)
    wts = torch.tensor(weights, **e.kw)
    g = torch.tensor(e.g, requires_grad=True, **e.kw)
    tau = torch.tensor(case["tau"], requires_grad=True, **e.kw)
    f0 = e.f.clone().requires_grad_(True)
    f, loss = f0, torch.zeros((), **e.kw)
    for t in range(case["steps"]):
        q = vel[t][at]
        v, w = [q[..., a] for a in range(3)], [q[..., 3 + a] for a in range(3)]
        up = [v[0] + (w[1] * d[2] - w[2] * d[1]), v[1] + (w[2] * d[0] - w[0] * d[2]),
              v[2] + (w[0] * d[1] - w[1] * d[0])]
        up = [torch.where(solid, c, torch.zeros_like(c)) for c in up]
        out, F = e.collide(f, up, 1.0 / tau, g)
        Fp, Tp = e.sums(F, owner, d, n)
        loss = loss + (wts[t, :, :3] * Fp).sum() + (wts[t, :, 3:] * Tp).sum()
        f = e.stream(out)
    loss.backward()
    res = {"loss": float(loss.detach()), "grad_vel": _rows(vel.grad.cpu(), _window_room(case), 1), "grad_body_force": g.grad.cpu(),
           "grad_tau": float(tau.grad)}
    if case["want_f0"]:
        res["grad_f0"] = f0.grad.cpu()
    return res
