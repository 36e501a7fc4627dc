"""The work that a user of this library has it do, as timed cases.

Every case is one of the library's public calls with the sizes it is used
at:

field   the velocity of all vortices of a body (convective velocity and
        3-nearest distance, vortex diffusion, wall diffusion: vx_stage), read
        into pinned host arrays as a program that saves or plots the field does;
steps   a run between two saved frames: the vortices in from pinned host
        arrays, whole time steps (vx_step), the vortices and forces out;
batch   the same for a population of bodies advanced together (vx_batch);
body    a body taken on: vx_create (profile up, panel system built and
        inverted) and the inverted panel system read back, as a server
        admitting a request or a parameter study over shapes does;
probe   the velocity at the points of a square grid (vx_probe);
dropin  one step through the reference's own entry points (vort_creation,
        Speed, Step of include/vortex_b200_unit1.h) on the caller's device
        records.

The vortices are the warm wake of vortex_b200.workloads behind a cylinder or
the rounded plate, and the seeded Gaussian clouds of its multi-body
population.  Results of the FP32 bulk form are kept as float32 (a saved frame
holds six decimals), those of the plain FP64 form as float64.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

from vortex_b200 import native as N
from vortex_b200 import profiles
from vortex_b200 import workloads as wl

BULK, PLAIN = "bulk", "plain"


def listed():
    return [
        # the smallest body of the multi-body population: launches and latency
        dict(name="field_1k", kind="field", form=BULK, panels=200, n=1000),
        # the 200-panel cylinder in its first hundreds of steps
        dict(name="field_30k", kind="field", form=BULK, panels=200, n=30_011),
        # a middle size of the 1000-panel cylinder
        dict(name="field_250k", kind="field", form=BULK, panels=1000, n=250_000),
        # the 1000-panel cylinder's wake at the benchmark's size
        dict(name="field_1m", kind="field", form=BULK, panels=1000, n=1_000_000),
        # the plain FP64 form, the one results are checked with
        dict(name="field_plain_12k", kind="field", form=PLAIN, panels=200, n=12_345),
        # a run of the 200-panel cylinder between two frames
        dict(name="steps_20k", kind="steps", form=BULK, body="circle", panels=200, n=20_000, steps=8),
        # the benchmark's body: 1000 panels, 1e6 vortices
        dict(name="steps_1m", kind="steps", form=BULK, body="circle", panels=1000, n=1_000_000, steps=4),
        # the largest configuration: the 2576-panel plate at 20 degrees
        dict(name="steps_plate_3m", kind="steps", form=BULK, body="plate", panels=2576, n=3_000_000, steps=2),
        # small and middle bodies of the population, batched
        dict(name="batch_16", kind="batch", bodies=16, n=20_000, steps=8),
        # a body of the benchmark's panel count taken on
        dict(name="body_1000", kind="body", panels=1000),
        # a 64 x 64 probe grid over the benchmark's wake
        dict(name="probe_64x64_1m", kind="probe", form=BULK, panels=200, n=1_000_000, side=64),
        # the reference's driver linked against this library, plain FP64
        dict(name="dropin_16k", kind="dropin", panels=200, n=16_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["field", "field", "field", "steps", "steps", "batch", "body", "probe", "dropin"])
    panels = _log_int(rng, 200, 1000)
    if kind == "field":
        if rng.random() < 0.25:
            return dict(kind=kind, form=PLAIN, panels=panels, n=_log_int(rng, 1000, 16_000))
        return dict(kind=kind, form=BULK, panels=panels, n=_log_int(rng, 1000, 1_000_000))
    if kind == "steps":
        n = _log_int(rng, 2000, 2_000_000)
        body = rng.choice(["circle", "ellipse", "plate"])
        return dict(kind=kind, form=BULK, body=body, panels=panels, n=n, steps=rng.randint(1, 8 if n < 200_000 else 4))
    if kind == "batch":
        return dict(kind=kind, bodies=rng.randint(4, 24), n=_log_int(rng, 2000, 20_000), steps=rng.randint(2, 8))
    if kind == "body":
        return dict(kind=kind, panels=_log_int(rng, 64, 1200))
    if kind == "probe":
        return dict(kind=kind, form=rng.choice([BULK, BULK, PLAIN]), panels=200, n=_log_int(rng, 1000, 200_000),
                    side=rng.randint(8, 64))
    return dict(kind=kind, panels=panels, n=_log_int(rng, 1000, 16_000))


def work(case):
    """Bytes: inputs once in, results once out.  Operations, per unit of pair
    work: 12 a Biot-Savart pair, 18 a diffusion pair.  The bulk form cannot do
    without its neighbour sums: about 970 diffusion pairs a vortex (a circle
    of 16 mean 3-nearest distances) and 288 near-field pairs (9 leaves of 32),
    and 27 x 16^2 complex products a leaf of 32 for the far field."""
    k = case["kind"]
    if k == "body":
        s = case["panels"] + 1
        return {"bytes": 120.0 * case["panels"] + 8.0 * s * s, "flops": 2.0 * s ** 3}
    n = float(case["n"])
    bulk = 970 * 18 + 288 * 12 + 27 * 256 * 8 / 32
    if k == "field":
        return {"bytes": 48.0 * n, "flops": n * (n * 30 if case["form"] == PLAIN else bulk)}
    if k == "probe":
        m = case["side"] ** 2
        return {"bytes": 24.0 * n + 32.0 * m, "flops": 12.0 * n * m}
    P = float(case.get("panels", 400))
    if k == "dropin":
        return {"bytes": 48.0 * n + 8 * (P + 1) ** 2, "flops": n * n * 30 + 30 * P * n + 2 * P * P}
    if k == "batch":
        n = sum(_batch_sizes(case))
    return {"bytes": 48.0 * n, "flops": case["steps"] * n * bulk}


# ---------------------------------------------------------------------------
# Bodies and vortices.
def _precision(case):
    return N.PREC_FP64 if case.get("form") == PLAIN else N.PREC_FP32


def _body(case, seed):
    """(configuration, panel records) of a single body."""
    P, prec = case["panels"], _precision(case)
    shape = case.get("body", "circle")
    if shape == "plate":
        pan = profiles.rotate(profiles.rounded_plate(P), -20.0)
        return N.default_conf(steps=5000, dt=0.001, viscosity=1e-4, v_inf_x=1.0, v_inf_y=0.0, x_min=-2.0, x_max=10.0,
                              y_min=-10.0, y_max=10.0, ve_size=float(np.mean(pan["length"])), n_of_points=20, n_col=2,
                              r_col_diff_sign=0.0, r_col_same_sign=0.3, max_ve_g=1e30, v_inf_incr_steps=0,
                              drop_eps=1e-8, birth_offset_mode=N.BIRTH_HALF_PANEL, precision=prec, inc_step=65536,
                              gj_pivot=2), pan
    if shape == "ellipse":
        pan = profiles.ellipse(P, 0.5, 0.05 + 0.45 * random.Random(seed).random())
        return wl.cylinder_conf(prec, P, ve_size=float(np.mean(pan["length"])), gj_pivot=2), pan
    return wl.cylinder_conf(prec, P), profiles.circle(P)


def _pinned(*arrays):
    return [torch.from_numpy(a).pin_memory() for a in arrays]


def _kept(case, *arrays):
    """Results as the form holds them."""
    return [a.clone() if case.get("form") == PLAIN else a.to(torch.float32) for a in arrays]


def _read_frame(sim, buffers):
    """The body's vortices into buffers that hold at least as many, zeros
    after them; their count."""
    m = sim.particles_into(*(t.numpy() for t in buffers))
    for t in buffers:
        t[m:] = 0.0
    return m


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _ok(rc):
    if rc != 0:
        raise N.VxError("call failed with %d (%s)" % (rc, N.lib().vx_last_error().decode()))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "body":
        b = 0.2 + 0.3 * random.Random(seed).random()
        pan = profiles.ellipse(case["panels"], 0.5, b)
        conf = wl.cylinder_conf(N.PREC_FP32, case["panels"], ve_size=float(np.mean(pan["length"])), gj_pivot=2)
        S = case["panels"] + 1
        return dict(case=case, conf=conf, pan=pan, out=torch.zeros(S, S, dtype=torch.float64).pin_memory())
    if kind == "batch":
        return _prepare_batch(case, seed)
    x, y, g = wl.warm_wake(case["n"], seed)
    if kind == "dropin":
        return _prepare_dropin(case, seed, x, y, g)
    conf, pan = _body(case, seed)
    sim = N.Sim(conf, pan)
    state = dict(case=case, sim=sim)
    if kind == "steps":
        room = case["n"] + case["steps"] * case["panels"]
        state["frame"] = [t.numpy() for t in _pinned(x, y, g)]
        state["out"] = _pinned(*(np.zeros(room) for _ in range(3)))
        sim.set_particles(*state["frame"])
        return state
    sim.set_particles(x, y, g)
    if kind == "probe":
        gx, gy = np.meshgrid(np.linspace(-1.0, 3.0, case["side"]), np.linspace(-1.0, 1.0, case["side"]), indexing="xy")
        state["points"] = (gx.ravel(), gy.ravel())
    else:
        state["out"] = _pinned(*(np.zeros(case["n"]) for _ in range(3)))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "field":
        sim = state["sim"]
        sim.stage("velocity", "diffusion", "wall")
        _ok(N.lib().vx_get_velocity(sim.h, *(_ptr(t) for t in state["out"]), C.c_int64(case["n"])))
        return dict(zip(("vx", "vy", "d"), _kept(case, *state["out"])))
    if kind == "steps":
        sim = state["sim"]
        sim.set_particles(*state["frame"])
        sim.set_dg(0.0)
        sim.step(case["steps"])
        m = _read_frame(sim, state["out"])
        out = dict(zip("xyg", _kept(case, *state["out"])))
        out["forces"] = _kept(case, torch.from_numpy(sim.forces()))[0]
        out["n"] = m
        return out
    if kind == "body":
        sim = N.Sim(state["conf"], state["pan"])
        _ok(N.lib().vx_get_matrix(sim.h, _ptr(state["out"])))
        sim.close()
        return state["out"]
    if kind == "probe":
        u, v = state["sim"].probe(*state["points"])
        return _kept(case, torch.from_numpy(u), torch.from_numpy(v))
    if kind == "batch":
        return _run_batch(state)
    return _run_dropin(state)


# ---------------------------------------------------------------------------
# A population of bodies: shapes, panel counts (200 to 800) and cloud sizes
# (1000 to n, log-uniform) fixed by the case, the clouds by the seed.
def _batch_sizes(case):
    r = random.Random(1000 * case["bodies"] + case["n"])
    return [_log_int(r, 1000, case["n"]) for _ in range(case["bodies"])]


def _prepare_batch(case, seed):
    r = random.Random(case["bodies"])
    sims, frames = [], []
    for k, n in enumerate(_batch_sizes(case)):
        P = _log_int(r, 200, 800)
        spec = wl.body_spec(7, k)
        spec.update(panels=P, dt=0.005 * 200.0 / P, n0=n, cloud_seed=int(wl.splitmix64(seed, 1, offset=k)[0]))
        conf, pan, x, y, g = wl.make_body(spec, N.PREC_FP32)
        sim = N.Sim(conf, pan)
        sim.set_particles(x, y, g)
        sims.append(sim)
        frames.append([t.numpy() for t in _pinned(x, y, g)])
    rooms = [len(f[0]) + case["steps"] * s.P for f, s in zip(frames, sims)]
    out = _pinned(*(np.zeros(sum(rooms)) for _ in range(3)))
    return dict(case=case, sims=sims, frames=frames, batch=N.Batch(sims), out=out,
                parts=list(zip(*(t.split(rooms) for t in out))))


def _run_batch(state):
    case, batch = state["case"], state["batch"]
    for sim, frame in zip(state["sims"], state["frames"]):
        sim.set_particles(*frame)
        sim.set_dg(0.0)
    batch.step(case["steps"])
    last = batch.last_results()
    for sim, part in zip(state["sims"], state["parts"]):
        _read_frame(sim, part)
    out = dict(zip("xyg", _kept(case, *state["out"])))
    rec = np.array([last[s.h.value] for s in state["sims"]])
    out["n"] = rec[:, 0].astype(np.int64)
    out["forces"] = rec[:, 1:].astype(np.float32)
    return out


# ---------------------------------------------------------------------------
# The reference's entry points on device records.
class _UnitConf(C.Structure):
    """struct vxu_conf_t of include/vortex_b200_unit1.h."""
    _fields_ = [
        ("steps", C.c_size_t), ("saving_step", C.c_size_t), ("dt", C.c_double), ("inc_step", C.c_size_t),
        ("viscosity", C.c_double), ("rho", C.c_double), ("v_inf_x", C.c_double), ("v_inf_y", C.c_double),
        ("n_of_points", C.c_size_t), ("x_max", C.c_double), ("x_min", C.c_double), ("y_max", C.c_double),
        ("y_min", C.c_double), ("profile_x_min", C.c_double), ("profile_x_max", C.c_double),
        ("profile_y_min", C.c_double), ("profile_y_max", C.c_double), ("ve_size", C.c_double),
        ("n_col", C.c_size_t), ("h_col_x", C.c_double), ("h_col_y", C.c_double), ("rc_x", C.c_double),
        ("rc_y", C.c_double), ("pr_file", C.c_char * 256), ("birth_quant", C.c_size_t),
        ("r_col_diff_sign", C.c_double), ("r_col_same_sign", C.c_double), ("matrix_load", C.c_uint8),
        ("v_inf_incr_steps", C.c_size_t), ("max_ve_g", C.c_double), ("log_file", C.c_char * 256),
        ("config_file", C.c_char * 256), ("log_level", C.c_uint8), ("timings_file", C.c_char * 256),
        ("kadr_file", C.c_char * 256), ("second_points_file", C.c_char * 256), ("rel_t", C.c_double),
        ("steady_flow", C.c_uint8), ("no_log_buf", C.c_uint8),
    ]


def _prepare_dropin(case, seed, x, y, g):
    P, n, L = case["panels"], case["n"], N.lib()
    P32 = -(-P // 32) * 32
    pan = profiles.circle(P)
    c = wl.cylinder_conf(N.PREC_FP64, P)
    sim = N.Sim(c, pan)
    matrix = np.zeros((P32 + 1, P32 + 1))
    matrix[:P + 1, :P + 1] = sim.matrix()
    sim.close()
    u = _UnitConf.in_dll(L, "conf")
    C.memset(C.addressof(u), 0, C.sizeof(u))
    for k in ("dt", "viscosity", "rho", "v_inf_x", "v_inf_y", "x_max", "x_min", "y_max", "y_min", "ve_size", "rc_x",
              "rc_y", "r_col_diff_sign", "r_col_same_sign", "max_ve_g", "n_of_points", "n_col", "inc_step"):
        setattr(u, k, getattr(c, k))
    u.profile_x_min, u.profile_x_max = pan["left"][:, 0].min(), pan["left"][:, 0].max()
    u.profile_y_min, u.profile_y_max = pan["left"][:, 1].min(), pan["left"][:, 1].max()
    u.birth_quant = P
    padded = np.zeros(P32, dtype=pan.dtype)
    padded[:P] = pan
    cap = -(-(n + P) // 32) * 32 + 64
    start = np.zeros((cap, 3))
    start[:, 0] = start[:, 1] = 4e5 + np.arange(cap)
    start[:n] = np.stack([x, y, g], axis=1)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    state = dict(case=case, P32=P32, start=dev(start), pos=dev(start.copy()), vel=dev(np.zeros((cap, 2))),
                 d=dev(np.zeros(cap)), vinf=dev(np.array([c.v_inf_x, c.v_inf_y])), sums=dev(np.zeros(4)),
                 matrix=dev(matrix), panels=dev(padded.view(np.uint8).copy()), nu=c.viscosity)
    _ok(L.init_device_conf_values())
    return state


def _run_dropin(state):
    L, P, n = N.lib(), state["case"]["panels"], state["case"]["n"]
    pos, vel, d, vinf, pan = (_ptr(state[k]) for k in ("pos", "vel", "d", "vinf", "panels"))
    sums = state["sums"]
    state["pos"].copy_(state["start"])
    sums.zero_()                                    # d_g, force (x, y), moment
    dg, force, moment = (C.c_void_p(sums.data_ptr() + 8 * k) for k in (0, 1, 3))
    _ok(L.vort_creation(pos, vinf, C.c_size_t(P), C.c_size_t(state["P32"]), C.c_size_t(n), _ptr(state["matrix"]), dg,
                        pan))
    m = n + P
    slots = -(-m // 32) * 32
    _ok(L.Speed(pos, vinf, C.c_size_t(slots), vel, d, C.c_double(state["nu"]), pan))
    count = C.c_size_t(m)
    _ok(L.Step(pos, vel, C.byref(count), C.c_size_t(slots), dg, force, moment, pan))
    return dict(n=int(count.value), pos=state["pos"][:m].clone(), vel=state["vel"][:m].clone(), d=state["d"][:m].clone(),
                sums=sums.clone())


# ---------------------------------------------------------------------------
# The same values in 64 bits, in plain torch.
def _induced(tx, ty, x, y, g, eps, vinf=(1.0, 0.0)):
    """Smoothed Biot-Savart velocity at the points (tx, ty)."""
    u, v = torch.empty_like(tx), torch.empty_like(ty)
    step = max(1, (1 << 27) // len(x))
    for a in range(0, len(tx), step):
        dx, dy = tx[a:a + step, None] - x, ty[a:a + step, None] - y
        w = g / (dx * dx + dy * dy).clamp_(min=eps * eps)
        u[a:a + step] = -(w * dy).sum(1) / (2 * math.pi) + vinf[0]
        v[a:a + step] = (w * dx).sum(1) / (2 * math.pi) + vinf[1]
    return u, v


def _diffused(x, y, g, eps, nu):
    """Mean distance to the 3 nearest vortices and the diffusive velocity."""
    n = len(x)
    d, u, v = torch.empty_like(x), torch.zeros_like(x), torch.zeros_like(x)
    step = max(1, (1 << 27) // n)
    for a in range(0, n, step):
        b = min(n, a + step)
        dx, dy = x[a:b, None] - x, y[a:b, None] - y
        r = (dx * dx + dy * dy).sqrt_()
        r[torch.arange(b - a, device=x.device), torch.arange(a, b, device=x.device)] = math.inf
        da = r.topk(3, dim=1, largest=False).values.mean(1)
        e = torch.where(r > 0.001 * eps, g * torch.exp(-r / da[:, None]), 0.0)
        i1 = e.sum(1)
        e /= r
        ok = i1.abs() > 1e-5
        q = torch.where(ok, nu / torch.where(ok, i1 * da, 1.0), 0.0)
        d[a:b], u[a:b], v[a:b] = da, q * (e * dx).sum(1), q * (e * dy).sum(1)
    return d, u, v


def _walled(x, y, d, pan, nu, points):
    """Diffusive velocity off the wall (no vortex here lies within a tenth of
    a panel length of a birth point)."""
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(x)  # noqa: E731
    birth, left, right, norm, ln = (t(pan[k]) for k in ("birth", "left", "right", "norm", "length"))
    u, v = torch.zeros_like(x), torch.zeros_like(x)
    box = 5 * ln.max()
    near = ((x > birth[:, 0].min() - box) & (x < birth[:, 0].max() + box) & (y > birth[:, 1].min() - box)
            & (y < birth[:, 1].max() + box)).nonzero().ravel()
    h = (torch.arange(points, device=x.device, dtype=x.dtype) + 0.5) / points
    for i in near.split(64):
        xi, yi, di = x[i, None, None], y[i, None, None], d[i, None, None]
        close = torch.hypot(x[i, None] - birth[:, 0], y[i, None] - birth[:, 1]) < 5 * ln
        ex = (xi - (left[:, 0, None] + h * (right - left)[:, 0, None])) / di
        ey = (yi - (left[:, 1, None] + h * (right - left)[:, 1, None])) / di
        r = torch.hypot(ex, ey)
        w = torch.exp(-r) * (ln / points)[:, None] * close[:, :, None]
        en = -(ex * norm[:, 0, None] + ey * norm[:, 1, None])
        i0 = 2 * math.pi * d[i] ** 2 - d[i] * (en / r ** 2 * (r + 1) * w).sum((1, 2))
        ws = w.sum(2)
        u[i], v[i] = nu * (ws @ norm[:, 0]) / i0, nu * (ws @ norm[:, 1]) / i0
    return u, v


def exact(case, seed):
    if case["kind"] not in ("field", "probe") or (case["kind"] == "field" and case["n"] > 400_000):
        return None
    conf, pan = _body(case, seed)
    x, y, g = (torch.from_numpy(a).cuda() for a in wl.warm_wake(case["n"], seed))
    vinf = (conf.v_inf_x, conf.v_inf_y)
    if case["kind"] == "probe":
        gx, gy = np.meshgrid(np.linspace(-1.0, 3.0, case["side"]), np.linspace(-1.0, 1.0, case["side"]), indexing="xy")
        tx, ty = torch.from_numpy(gx.ravel()).cuda(), torch.from_numpy(gy.ravel()).cuda()
        return list(_induced(tx, ty, x, y, g, conf.ve_size, vinf))
    u, v = _induced(x, y, x, y, g, conf.ve_size, vinf)
    d, du, dv = _diffused(x, y, g, conf.ve_size, conf.viscosity)
    wu, wv = _walled(x, y, d, pan, conf.viscosity, conf.n_of_points)
    return dict(vx=u + du + wu, vy=v + dv + wv, d=d)
