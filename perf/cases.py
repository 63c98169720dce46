"""Work that users of this engine have it do, as cases that can be timed.

Each case is one pass of a user's loop through the public Python surface
(``lbm_ddf_b200``), whose calls are the C ABI's one to one:

* ``log``      march a resident case, then read Nu / KE / Re and, where a run
               writes it, the vertical profile (the driver's output events);
* ``observe``  march a resident case with the observables of every step;
* ``new_run``  start from a temperature field in page-locked host memory,
               march with the observables of every step, read the final ones;
* ``resume``   bring an evicted case back from its checkpoint, march it, evict
               it again (checkpoints in page-locked host memory);
* ``restart``  the reference's restart pair: load its FP64 fields, march,
               store them (pageable host arrays, as files are read and written);
* ``ensemble`` many resident cases, each on its own kernel (the launch the
               autotuner picks for ensembles), then every member's observables;
* ``serve``    one chunk of the serving loop: the tile-walk launch, then every
               member's observables through one asynchronous copy.

Results are handed on in the type of the populations they come from.
"""
import ctypes
import math
import random

import numpy as np
import torch

import lbm_ddf_b200 as lbm

Q = 27
CX = (0, 1, 0, -1, 0, 0, 0, 1, -1, -1, 1, 1, 0, -1, 0, 1, 0, -1, 0, 1, -1, -1, 1, 1, -1, -1, 1)
CY = (0, 0, 1, 0, -1, 0, 0, 1, 1, -1, -1, 0, 1, 0, -1, 0, 1, 0, -1, 1, 1, -1, -1, 1, 1, -1, -1)
CZ = (0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, 1, 1, -1, -1, -1, -1, 1, 1, 1, 1, -1, -1, -1, -1)
W = (8 / 27,) + (2 / 27,) * 6 + (1 / 54,) * 12 + (1 / 216,) * 8
OPP = tuple(next(j for j in range(Q) if (CX[j], CY[j], CZ[j]) == (-CX[i], -CY[i], -CZ[i])) for i in range(Q))

BYTES = {"f64": 8, "f32": 4, "f16s": 2, "bf16s": 2}
TYPES = {"f64": torch.float64, "f32": torch.float32, "f16s": torch.float16, "bf16s": torch.bfloat16}
# arithmetic (and carried-temperature) type
ARITH = {"f64": torch.float64, "f32": torch.float32, "f16s": torch.float32, "bf16s": torch.float32}

# the grids of the ensemble configuration, (x, vertical, z)
ENSEMBLE_GRIDS = ((32, 32, 32), (48, 48, 48), (64, 64, 64), (96, 96, 96), (128, 128, 128), (128, 64, 128),
                  (192, 96, 192))


def _case(kind, lx, ly, lz, storage, sides="periodic", collision="bgk", ra=1e6, pr=0.71, steps=100, **more):
    return dict(kind=kind, lx=lx, ly=ly, lz=lz, storage=storage, sides=sides, collision=collision, ra=ra, pr=pr,
                steps=steps, **more)


def _mix(kind, members, storage, mix, collision="bgk", steps=100):
    return dict(kind=kind, members=members, storage=storage, mix=mix, collision=collision, steps=steps)


def listed():
    named = {
        # a live display of the smallest ensemble grid: one step, one read
        "watch_f32_32": _case("log", 32, 32, 32, "f32", ra=3e4, steps=1, profile=False),
        # the FP64 validation run: 64^3, Nu and KE every 100 steps
        "nu_log_f64_64": _case("log", 64, 64, 64, "f64", ra=1e5, steps=100, profile=False),
        # the benchmark's new run: 256^3 closed box in FP64, every step's observables
        "new_run_f64_box_256": _case("new_run", 256, 256, 256, "f64", "wall", ra=1e7, steps=20),
        # the single-instance configuration in FP32, with the outputs of an output event
        "log_f32_256": _case("log", 256, 256, 256, "f32", ra=1e7, steps=100, profile=True),
        # a closed box of odd sizes: rows that do not fill warps
        "log_f32_box_ragged": _case("log", 201, 101, 151, "f32", "wall", ra=1e6, steps=50, profile=True),
        # the precision study's grid, the largest resident state of 16-bit storage here
        "precision_f16s_512": _case("log", 512, 256, 512, "f16s", ra=1e8, steps=20, profile=True),
        # a Nu time series at every step, closed box, BF16
        "observe_bf16s_box": _case("observe", 192, 96, 192, "bf16s", "wall", ra=1e6, steps=50),
        # a served case evicted from HBM and brought back, regularised collision
        "resume_f16s_reg": _case("resume", 128, 64, 128, "f16s", collision="regularized", ra=1e7, steps=200),
        # a run continued from the reference's restart files
        "restart_f64_box_64": _case("restart", 64, 64, 64, "f64", "wall", ra=1e5, steps=1000),
        # a third of the ensemble configuration between two Nu samples
        "ensemble_f16s": _mix("ensemble", 32, "f16s", mix=2024),
        # a chunk of the serving loop per storage format; under-resolved
        # requests are served with the regularised collision
        "serve_f32": _mix("serve", 16, "f32", mix=7),
        "serve_f16s_reg": _mix("serve", 16, "f16s", mix=8, collision="regularized"),
    }
    return [dict(c, name=n) for n, c in named.items()]


def draw(rng):
    kind = rng.choice(("log", "log", "observe", "new_run", "resume", "restart", "ensemble", "serve"))
    storage = rng.choice(tuple(BYTES))
    collision = rng.choice(("bgk", "bgk", "bgk", "regularized"))
    if kind in ("ensemble", "serve"):
        return _mix(kind, rng.randint(2, 24), storage, rng.randint(1, 10 ** 6), collision, rng.randint(10, 50))
    if kind == "restart":
        storage = "f64"

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    top = 96 if kind == "restart" else 320
    lx, ly, lz = size(24, top), size(24, min(top, 256)), size(24, top)
    ra = 1e5 * (ly / 48.0) ** 2 * 10 ** rng.uniform(-1, 0)
    steps = size(1, max(1, min(200, int(2e9 / (lx * ly * lz * BYTES[storage] / 8)))))
    if kind == "resume":
        steps += steps % 2
    c = _case(kind, lx, ly, lz, storage, rng.choice(("periodic", "wall")), collision, round(ra, 1),
              rng.choice((0.71, 4.38)), steps)
    if kind == "log":
        c["profile"] = rng.random() < 0.5
    return c


def _members(case):
    """The cases of an ensemble or serving mix (their grids and parameters
    belong to the case, their initial states to the seed)."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["members"]):
        if case["kind"] == "ensemble":
            lx, ly, lz = r.choice(ENSEMBLE_GRIDS)
            ra, pr = 1e5 * (ly / 48.0) ** 2 * 10 ** r.uniform(-1, 0), r.choice((0.71, 4.38, 7.0))
        else:   # horizontal size 48 to 192, aspect ratio 1 to 2
            lx = lz = int(round(r.uniform(48, 192) / 16)) * 16
            ly = max(16, int(round(lx / r.uniform(1, 2) / 8)) * 8)
            ra, pr = 1e5 * (ly / 48.0) ** 2 * 10 ** r.uniform(-1, 0), r.choice((0.71, 4.38))
        out.append(_case(case["kind"], lx, ly, lz, case["storage"], "periodic", case["collision"], ra, pr,
                         case["steps"]))
    return out


def _params(c):
    return lbm.make_params(c["lx"], c["ly"], c["lz"], rayleigh=c["ra"], prandtl=c["pr"], storage=c["storage"],
                           sides=lbm.SIDES_WALL if c["sides"] == "wall" else lbm.SIDES_PERIODIC)


def _nodes(c):
    return c["lx"] * c["ly"] * c["lz"]


def _grid(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = random.Random(seed)
    z = torch.arange(c["lz"], device="cuda", dtype=torch.float64)[:, None, None]
    y = torch.arange(c["ly"], device="cuda", dtype=torch.float64)[None, :, None]
    x = torch.arange(c["lx"], device="cuda", dtype=torch.float64)[None, None, :]
    return g, r, z, y, x


def _temperature(c, seed):
    """[lz, ly, lx] FP64: the conduction profile, convection rolls of random
    strength and phase, and the configurations' noise of 1e-3."""
    g, r, z, y, x = _grid(c, seed)
    t = 1.0 - y / (c["ly"] - 1.0) + torch.zeros_like(z) + torch.zeros_like(x)
    env = torch.sin(math.pi * (y + 0.5) / c["ly"])
    t += r.uniform(0.05, 0.15) * env * torch.cos(2 * math.pi * (x / c["lx"] + r.random()))
    t += r.uniform(0.05, 0.15) * env * torch.cos(2 * math.pi * (z / c["lz"] + r.random()))
    t += 1e-3 * (2.0 * torch.rand(t.shape, generator=g, device="cuda", dtype=torch.float64) - 1.0)
    return t


def _beta(c):
    return 0.01 / c["ly"]   # free-fall velocity 0.1, as make_params has it


def _flowing_state(c, seed):
    """A state in motion: f, g [27, lz, ly, lx], the previous step's
    temperature, all FP64."""
    g, r, z, y, x = _grid(c, seed + 1)
    phi = _temperature(c, seed)
    a = r.uniform(0.01, 0.04)
    kx, kz, ky = 2 * math.pi / c["lx"], 2 * math.pi / c["lz"], math.pi / c["ly"]
    wall = torch.sin(ky * (y + 0.5))
    ux = a * wall * torch.sin(kx * x + r.random()) * torch.cos(kz * z)
    uy = a * wall * torch.cos(kx * x) * torch.cos(kz * z + r.random())
    uz = a * wall * torch.cos(kx * x + r.random()) * torch.sin(kz * z)
    rho = 1e-3 * torch.cos(kx * x) * wall * torch.ones_like(z)
    f = torch.empty((Q,) + tuple(phi.shape), dtype=torch.float64, device="cuda")
    h = torch.empty_like(f)
    uu = ux * ux + uy * uy + uz * uz
    for k in range(Q):
        eu = 3.0 * (CX[k] * ux + CY[k] * uy + CZ[k] * uz)
        p = eu + 0.5 * eu * eu - 1.5 * uu
        n = 1.0 + 1e-2 * torch.rand(phi.shape, generator=g, device="cuda", dtype=torch.float64)
        f[k] = W[k] * (rho + p) * n
        h[k] = W[k] * phi * (1.0 + p) * n
    prev = phi + 1e-4 * torch.rand(phi.shape, generator=g, device="cuda", dtype=torch.float64)
    return f, h, prev


# ---- checkpoints (the native image: header, f, g, carried temperature) ------

def _row(c):
    return -(-_nodes(c) // 128) * 128


def _image_parts(c):
    """Offsets and bytes of the image: (header, populations, carried, total)."""
    pop = 2 * Q * _row(c) * BYTES[c["storage"]]
    return 256, pop, _row(c) * (8 if c["storage"] == "f64" else 4)


def _image_views(c, buf):
    """The populations and the carried temperature of an image, by node:
    FP64 / FP32 [2, 27, N]; 16-bit pairs [27, N, 2]."""
    hb, pop, carry = _image_parts(c)
    n = _nodes(c)
    v = buf[hb:hb + pop].view(TYPES[c["storage"]])
    v = v.view(Q, _row(c), 2)[:, :n] if BYTES[c["storage"]] == 2 else v.view(2, Q, _row(c))[:, :, :n]
    return v, buf[hb + pop:hb + pop + carry].view(ARITH[c["storage"]])[:n]


class _Header(ctypes.Structure):
    _fields_ = [("magic", ctypes.c_char * 8), ("p", lbm.LbmParams), ("step", ctypes.c_int64),
                ("swapped", ctypes.c_int32), ("flags", ctypes.c_int32), ("ps", ctypes.c_int64)]


def _shift(c):
    """The conduction profile that 16-bit storage keeps g relative to."""
    y = torch.arange(c["ly"], device="cuda", dtype=torch.float64)
    return (1.0 - (y + 0.5) / c["ly"])[None, :, None]


def _checkpoint(c, seed):
    """A checkpoint of a flowing state in page-locked memory."""
    f, g, prev = _flowing_state(c, seed)
    buf = torch.zeros(sum(_image_parts(c)), dtype=torch.uint8, pin_memory=True)
    h = _Header(magic=b"LBMDDF3", p=_params(c), step=0, swapped=0, flags=0, ps=_row(c))
    buf[:ctypes.sizeof(h)] = torch.frombuffer(bytearray(bytes(h)), dtype=torch.uint8)
    pops, carried = _image_views(c, buf)
    n, t = _nodes(c), TYPES[c["storage"]]
    for k in range(Q):
        if BYTES[c["storage"]] == 2:
            pair = torch.stack(((f[k] / W[k]).view(n), (g[k] / W[k] - _shift(c)).reshape(n)), 1)
            pops[k].copy_(pair.to(t))
        else:
            pops[0, k].copy_(f[k].view(n).to(t))
            pops[1, k].copy_(g[k].view(n).to(t))
    carried.copy_(prev.view(n).to(ARITH[c["storage"]]))
    return buf


# ---- a pass -----------------------------------------------------------------

def _make(c):
    e = lbm.Case(_params(c))
    e.set_collision(c["collision"])
    return e


def _start(c, seed):
    e = _make(c)
    e.init_temperature(_temperature(c, seed).to(ARITH[c["storage"]]).contiguous())
    return e


def _table(storage, records):
    """Records of observables as tensors: the velocity beside its own scale."""
    t = TYPES[storage]
    nu = [[o["nu_bulk"], o["nu_top"], o["nu_bottom"]] for o in records]
    re = [[o["re"]] for o in records]
    u = [[math.sqrt(2.0 * o["ke"]), o["ux_mean"], o["uy_mean"], o["uz_mean"]] for o in records]
    phi = [[o["phi_mean"]] for o in records]
    steps = [[o["step"], o["diverged"]] for o in records]
    return {"nu": torch.tensor(nu, dtype=torch.float64).to(t), "re": torch.tensor(re, dtype=torch.float64).to(t),
            "velocity": torch.tensor(u, dtype=torch.float64).to(t),
            "phi": torch.tensor(phi, dtype=torch.float64).to(t), "steps": torch.tensor(steps)}


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("log", "observe"):
        s["engine"] = _start(case, seed)
    elif kind == "new_run":
        s["engine"] = _make(case)
        t = _temperature(case, seed).to(ARITH[case["storage"]])
        s["temperature"] = torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)
    elif kind == "resume":
        s["engine"] = _make(case)
        s["image"] = _checkpoint(case, seed)
        s["out"] = torch.empty_like(s["image"], pin_memory=True)
    elif kind == "restart":
        s["engine"] = _make(case)
        f, g, prev = _flowing_state(case, seed)
        m = _moments(case, f, g, prev)
        s["fields"] = [a.cpu().numpy() for a in (*m, f, g)]
    else:
        s["stream"] = torch.cuda.Stream()
        s["engines"] = [_start(c, seed * 1000 + i) for i, c in enumerate(_members(case))]
        s["batch"] = lbm.Batch(case["storage"])
        if kind == "ensemble":
            s["batch"].set_launch("per_case")
        for e in s["engines"]:
            s["batch"].add(e)
        s["buffer"] = lbm.ObservablesBuffer(len(s["engines"]))
        torch.cuda.synchronize()
    return s


def run(s):
    c, kind = s["case"], s["kind"]
    if kind == "log":
        e = s["engine"]
        e.step(c["steps"])
        out = _table(c["storage"], [e.observables()])
        if c["profile"]:
            out["profile"] = torch.from_numpy(e.profile()).to(TYPES[c["storage"]])
        return out
    if kind == "observe":
        return _table(c["storage"], s["engine"].step_observed(c["steps"]))
    if kind == "new_run":
        e = s["engine"]
        e.init_temperature(s["temperature"])
        return _table(c["storage"], e.step_observed(c["steps"]) + [e.observables()])
    if kind == "resume":
        e = s["engine"]
        e.restore_state(s["image"])
        e.step(c["steps"])
        e.save_state(s["out"])
        pops, carried = _image_views(c, s["out"])
        return {"header": s["out"][:ctypes.sizeof(_Header)], "populations": pops, "carried": carried}
    if kind == "restart":
        e = s["engine"]
        e.load_ref_state(*s["fields"])
        e.step(c["steps"])
        return e.store_ref_state()
    b = s["batch"]
    b.step(c["steps"], stream=s["stream"])
    if kind == "ensemble":
        return _table(c["storage"], b.observables(stream=s["stream"]))
    b.observables_async(s["buffer"], stream=s["stream"])
    s["stream"].synchronize()
    return _table(c["storage"], [s["buffer"][i] for i in range(len(s["engines"]))])


def work(case):
    """Every step reads and writes the state once; outputs that read the
    state do so once; what crosses to or from the host is counted on both
    sides."""
    kind = case["kind"]
    total = {"bytes": 0.0, "flops": 0.0}
    for c in _members(case) if kind in ("ensemble", "serve") else [case]:
        b, n = BYTES[c["storage"]], _nodes(c)
        carry = 8 if b == 8 else 4
        state = n * (2 * Q * b + carry)
        moved = 2.0 * state * c["steps"]
        if kind in ("log", "ensemble", "serve"):
            moved += state
        elif kind == "new_run":
            moved += 2 * state + n * carry
        elif kind == "resume":
            moved += 4 * state
        elif kind == "restart":
            moved += 2 * (state + n * 8 * (2 * Q + 5))
        total["bytes"] += moved
        total["flops"] += 800.0 * n * c["steps"]   # moments 6, equilibrium and relaxation 8 or 9 per population
    return total


# ---- the same in 64 bits, in plain torch ------------------------------------

def _derived(c):
    gb = _beta(c)
    visc = c["ly"] * math.sqrt(gb * c["ly"] * c["pr"] / c["ra"])
    diff = visc / c["pr"]
    return gb, visc, diff, 3.0 * visc + 0.5, 3.0 * diff + 0.5


def _moments(c, f, g, prev):
    rho = f.sum(0)
    ux = sum(CX[k] * f[k] for k in range(Q) if CX[k])
    uy = sum(CY[k] * f[k] for k in range(Q) if CY[k]) + 0.5 * _beta(c) * (prev - 0.5)
    uz = sum(CZ[k] * f[k] for k in range(Q) if CZ[k])
    return rho, ux, uy, uz, g.sum(0)


def _face(c, k, axis):
    """The index of the nodes whose population k came through a wall of
    `axis` (0 z, 1 y, 2 x), or None."""
    d = (CZ, CY, CX)[axis][k]
    if d == 0:
        return None
    at = [slice(None)] * 3
    at[axis] = 0 if d > 0 else (c["lz"], c["ly"], c["lx"])[axis] - 1
    return tuple(at)


def _exact_step(c, f, g, f2, g2, prev):
    """One step from (f, g, prev) into (f2, g2); returns phi, the next prev."""
    gb, _, _, tau, tauc = _derived(c)
    rho, ux, uy, uz, phi = _moments(c, f, g, prev)
    uu = 1.5 * (ux * ux + uy * uy + uz * uz)
    kf = 3.0 * (1.0 - 0.5 / tau) * gb * (phi - 0.5)
    if c["collision"] == "regularized":
        pi, j = {}, []
        u = (ux, uy, uz)
        for a in range(3):
            for b in range(a, 3):
                pi[a, b] = sum((CX, CY, CZ)[a][k] * (CX, CY, CZ)[b][k] * f[k] for k in range(Q)
                               if (CX, CY, CZ)[a][k] * (CX, CY, CZ)[b][k]) - u[a] * u[b]
                if a == b:
                    pi[a, b] = pi[a, b] - rho / 3.0
            j.append(sum((CX, CY, CZ)[a][k] * g[k] for k in range(Q) if (CX, CY, CZ)[a][k]) - phi * u[a])
        tr = (pi[0, 0] + pi[1, 1] + pi[2, 2]) / 3.0
    for k in range(Q):
        eu = 3.0 * (CX[k] * ux + CY[k] * uy + CZ[k] * uz) if k else torch.zeros_like(ux)
        p = eu + 0.5 * eu * eu - uu
        force = kf * (CY[k] - uy) * (W[k] * (1.0 + p))
        if c["collision"] == "regularized":
            ck = (CX[k], CY[k], CZ[k])
            q = -tr + sum((1 if a == b else 2) * ck[a] * ck[b] * pi[a, b] for a in range(3) for b in range(a, 3)
                          if ck[a] * ck[b])
            f[k] = W[k] * (rho + p) + (1.0 - 1.0 / tau) * 4.5 * W[k] * q + force
            cj = sum(ck[a] * j[a] for a in range(3) if ck[a]) if k else 0.0
            g[k] = W[k] * phi * (1.0 + p) + (1.0 - 1.0 / tauc) * 3.0 * W[k] * cj
        else:
            f[k] += force - (f[k] - W[k] * (rho + p)) / tau
            g[k] -= (g[k] - W[k] * phi * (1.0 + p)) / tauc
    for k in range(Q):
        shift = (CZ[k], CY[k], CX[k])
        o = OPP[k]
        f2[k] = torch.roll(f[k], shift, (0, 1, 2))
        g2[k] = torch.roll(g[k], shift, (0, 1, 2))
        # walls in the order x, y, z: the last rule at an edge holds
        for axis in (2, 1, 0) if c["sides"] == "wall" else (1,):
            at = _face(c, k, axis)
            if at is None:
                continue
            f2[k][at] = f[o][at]
            g2[k][at] = g[o][at]
            if axis == 1:
                g2[k][at] = 2.0 * W[k] * (1.0 if CY[k] > 0 else 0.0) * (1.0 + rho[at]) - g[o][at]
    return phi


def _exact_march(c, f, g, prev, steps, each=None):
    f2, g2 = torch.empty_like(f), torch.empty_like(g)
    for _ in range(steps):
        if each is not None:
            each(f, g, prev)
        prev = _exact_step(c, f, g, f2, g2, prev)
        f, f2, g, g2 = f2, f, g2, g
    return f, g, prev


def _exact_start(c, seed):
    t = _temperature(c, seed).to(ARITH[c["storage"]]).double()
    g = torch.stack([W[k] * t for k in range(Q)])
    return torch.zeros_like(g), g, t


def _exact_record(c, step, f, g, prev):
    _, visc, diff, _, _ = _derived(c)
    _, ux, uy, uz, phi = _moments(c, f, g, prev)
    ke = 0.5 * (ux * ux + uy * uy + uz * uz).mean().item()
    t = phi.mean((0, 2)).tolist()
    ly = c["ly"]
    return dict(step=step, diverged=0, nu_bulk=1.0 + (uy * phi).mean().item() * ly / diff,
                nu_top=-(3 * t[-1] - 4 * t[-2] + t[-3]) / 2 * ly,
                nu_bottom=-(-3 * t[0] + 4 * t[1] - t[2]) / 2 * ly, ke=ke, re=math.sqrt(2 * ke) * ly / visc,
                ux_mean=ux.mean().item(), uy_mean=uy.mean().item(), uz_mean=uz.mean().item(),
                phi_mean=phi.mean().item())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ensemble", "serve"):
        records = []
        for i, c in enumerate(_members(case)):
            state = _exact_march(c, *_exact_start(c, seed * 1000 + i), c["steps"])
            records.append(_exact_record(c, c["steps"], *state))
        return _table("f64", records)
    steps = case["steps"]
    if kind in ("log", "observe", "new_run"):
        records = []

        def each(*state):
            records.append(_exact_record(case, len(records), *state))

        state = _exact_march(case, *_exact_start(case, seed), steps, None if kind == "log" else each)
        if kind != "observe":
            records.append(_exact_record(case, steps, *state))
        out = _table("f64", records)
        if kind == "log" and case["profile"]:
            _, ux, uy, uz, phi = _moments(case, *state)
            p = phi.mean((0, 2))
            rms = ((phi - p[None, :, None]) ** 2).mean((0, 2)).sqrt()
            out["profile"] = torch.stack([a.mean((0, 2)) for a in (ux, uy, uz)] + [p, rms], 1).cpu()
        return out
    if kind == "restart":
        f, g, prev = _exact_march(case, *_flowing_state(case, seed), steps)
        names = ("rho", "ux", "uy", "uz", "phi", "f", "g")
        return {k: a.cpu().numpy() for k, a in zip(names, (*_moments(case, f, g, prev), f, g))}
    pops, carried = (a.cuda().double() for a in _image_views(case, _checkpoint(case, seed)))
    shape = (Q, case["lz"], case["ly"], case["lx"])
    w = torch.tensor(W, dtype=torch.float64, device="cuda").view(Q, 1, 1, 1)
    short = BYTES[case["storage"]] == 2
    if short:
        f, g = pops[..., 0].reshape(shape) * w, (pops[..., 1].reshape(shape) + _shift(case)) * w
    else:
        f, g = pops[0].reshape(shape).clone(), pops[1].reshape(shape).clone()
    f, g, prev = _exact_march(case, f, g, carried.reshape(shape[1:]), steps)
    if short:
        pops = torch.stack(((f / w).view(Q, -1), (g / w - _shift(case)).reshape(Q, -1)), 2)
    else:
        pops = torch.stack((f.view(Q, -1), g.view(Q, -1)))
    return {"header": None, "populations": pops, "carried": prev.reshape(-1)}
