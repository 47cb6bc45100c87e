"""The work that a user of this engine has it do, as cases that can be timed and compared.

A case is one call, or one short stretch of a run, through the public entry points (the C ABI by way of
``ncorpion_b200.api``):

* ``field``    one force evaluation of every body: on device buffers (an integrator of the caller's own, one
  call a kick) or on host buffers (a C host that keeps its arrays), in the three arithmetic modes;
* ``bf``       steps of the brute-force driver: gravity, collision search with mergers or rebounds, end of step;
* ``mesh``     steps of the mesh driver, in its order-free and its bit-exact modes, with and without the central
  body's J2 and tides;
* ``hybrid``   mesh collisions with fragmentation and brute-force gravity over every body;
* ``output``   an output step's cartesian files and statistics;
* ``forward`` / ``adjoint``  the differentiable leapfrog: final state, or that and the gradients.

The stepping cases upload a state, advance it and read it back, which is what a run between two outputs does.
"""
import ctypes as C

import numpy as np
import torch

from ncorpion_b200 import api

CENTRAL = (0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0, 1.0)  # the central body: at rest, mass 1, radius 1
CUBE_MIN = 4.4                                      # smallest collision cube: holds disks out to 2.2
NEIGHBOURS = 16.0                                   # neighbours a body is meant to have in the mesh
SOFTENING = 0.5


# ------------------------------------------------------------------- cases --

def listed():
    return [
        # a small run's kick by a C host that keeps its own arrays: latency and launches
        dict(name="field_exact_host_1000", kind="field", mode="exact", n=1000, radii="equal", soft=True, holes=0.0, host=True),
        # the drop-in's default arithmetic on a population of ordinary size
        dict(name="field_exact_20011", kind="field", mode="exact", n=20011, radii="equal", soft=True, holes=0.0, host=False),
        # full precision without the reference's order; slots emptied by earlier mergers
        dict(name="field_fp64_30011", kind="field", mode="fp64", n=30011, radii="equal", soft=False, holes=0.1, host=False),
        # small mixed call, radii of a size distribution, host buffers, empty slots
        dict(name="field_mixed_host_12345", kind="field", mode="mixed", n=12345, radii="law", soft=True, holes=0.05, host=True),
        # the headline of bench.py
        dict(name="field_mixed_65536", kind="field", mode="mixed", n=65536, radii="equal", soft=True, holes=0.0, host=False),
        # the gravity of the fragmenting disk's size, no softening
        dict(name="field_mixed_262144", kind="field", mode="mixed", n=262144, radii="law", soft=False, holes=0.0, host=False),
        # the collisional disk of bench.py
        dict(name="bf_merge_2000", kind="bf", n=2000, steps=20, treat="merge"),
        # the mesh disk of bench.py at full size
        dict(name="mesh_fast_1048576", kind="mesh", mode="mixed", n=1048576, steps=10, central="plain"),
        # a whole program's size in the drop-in's bit-exact arithmetic, with the central body's bulge and tides
        dict(name="mesh_exact_20011", kind="mesh", mode="exact", n=20011, steps=10, central="j2_tides"),
        # an output step's files
        dict(name="output_200000", kind="output", n=200000),
        # a gradient through one checkpoint segment of the differentiable disk of bench.py
        dict(name="adjoint_mixed_16384", kind="adjoint", mode="mixed", n=16384, steps=32),
        # the same in full precision, a smaller odd population
        dict(name="adjoint_fp64_5003", kind="adjoint", mode="exact", n=5003, steps=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["field"] * 5 + ["adjoint"] * 2 + ["mesh"] * 2 + ["forward", "bf", "hybrid", "output"])
    if kind == "field":
        mode = rng.choice(["exact", "fp64", "mixed", "mixed"])
        n = _log_int(rng, 200, {"exact": 50000, "fp64": 100000, "mixed": 250000}[mode])
        return dict(kind=kind, mode=mode, n=n, radii=rng.choice(["equal", "law"]), soft=rng.random() < 0.6,
                    holes=rng.choice([0.0, 0.0, 0.03, 0.25]), host=rng.random() < 0.3)
    if kind == "bf":
        return dict(kind=kind, n=_log_int(rng, 100, 4000), steps=20, treat=rng.choice(["merge", "inelastic"]))
    if kind == "mesh":
        mode = rng.choice(["mixed", "mixed", "exact"])
        n = _log_int(rng, 5000, 1000000 if mode == "mixed" else 100000)
        return dict(kind=kind, mode=mode, n=n, steps=rng.randint(5, 10), central=rng.choice(["plain", "plain", "j2", "j2_tides"]))
    if kind == "hybrid":
        return dict(kind=kind, mode=rng.choice(["mixed", "fp64"]), n=_log_int(rng, 5000, 100000), steps=2)
    if kind == "output":
        return dict(kind=kind, n=_log_int(rng, 1000, 500000))
    mode = rng.choice(["mixed", "exact"])
    return dict(kind=kind, mode=mode, n=_log_int(rng, 300, 16000 if mode == "mixed" else 9000), steps=rng.randint(4, 32))


# ------------------------------------------------------------------ inputs --

def _disk(rng, n, a_lo, a_hi, sig_e, sig_i, mass, radius):
    """Bodies on Kepler orbits about a unit mass: semi-major axes uniform, eccentricities and inclinations Rayleigh."""
    a = rng.uniform(a_lo, a_hi, n)
    e = np.minimum(rng.rayleigh(sig_e, n), 0.9)
    inc = rng.rayleigh(sig_i, n)
    nu, om, node = rng.uniform(0.0, 2.0 * np.pi, (3, n))
    p = a * (1.0 - e * e)
    r, s = p / (1.0 + e * np.cos(nu)), np.sqrt((1.0 + mass) / p)
    ca, sa, co, so = np.cos(om + nu), np.sin(om + nu), np.cos(om), np.sin(om)
    u, w = r * ca, r * sa
    vu, vw = -s * (sa + e * so), s * (ca + e * co)
    cn, sn, ci, si = np.cos(node), np.sin(node), np.cos(inc), np.sin(inc)
    b = np.empty((n, 8))
    for c, (f, g) in enumerate(((u, w), (vu, vw))):
        b[:, 3 * c] = cn * f - sn * ci * g
        b[:, 3 * c + 1] = sn * f + cn * ci * g
        b[:, 3 * c + 2] = si * g
    b[:, 6], b[:, 7] = mass, radius
    return b


def _size_law(rng, n, lo, hi):
    """Radii of dN/dR ~ R^-3.5 over [lo, hi]."""
    return (lo ** -2.5 + rng.random(n) * (hi ** -2.5 - lo ** -2.5)) ** (1.0 / -2.5)


def _bodies(case, seed):
    rng = np.random.default_rng([seed, case["n"]])
    n, kind = case["n"], case["kind"]
    if kind == "bf":
        return _disk(rng, n, 0.8, 1.2, 0.01, 0.005, np.full(n, 1e-3 / n), np.full(n, 2e-3))
    if kind in ("mesh", "output"):
        rad = _size_law(rng, n, 1e-5, 1e-3)
        return _disk(rng, n, 0.5, 2.0, 0.01, 0.005, 4.0 * np.pi * rad ** 3, rad)
    if kind == "hybrid":
        rad = rng.uniform(2e-4, 5e-4, n)
        return _disk(rng, n, 0.9, 1.1, 0.02, 0.02, 4.0 * np.pi * rad ** 3, rad)
    rad = 1e-2 if kind in ("adjoint", "forward") else 1e-5
    rad = _size_law(rng, n, 1e-5, 1e-3) if case.get("radii") == "law" else np.full(n, rad)
    return _disk(rng, n, 0.8, 1.2, 0.01, 0.005, 10.0 ** rng.uniform(-9.0, -6.0, n), rad)


def _exists(case, seed):
    ex = np.ones(case["n"], np.int32)
    ex[np.random.default_rng([seed, 1]).random(case["n"]) < case.get("holes", 0.0)] = 0
    return ex


def _params(case):
    kind = case["kind"]
    p = dict(G=1.0, softening_parameter=0.0, collision_bool=0, disruption_threshold=0.1, high_dumping_threshold=100.0,
             gravity_mode=api.GRAVITY_MODES[case.get("mode", "exact")])
    if kind == "field":
        p.update(softening_parameter=SOFTENING if case["soft"] else 0.0)
    elif kind in ("adjoint", "forward"):
        p.update(softening_parameter=SOFTENING)
    elif kind == "bf":
        p.update(collision_bool=1, collision_type=api.COLLISION_MERGER if case["treat"] == "merge" else api.COLLISION_INELASTIC)
    else:
        p.update(collision_bool=1, brute_force_bool=0, mesh_bool=1, collision_cube_cells=_cells(case["n"]),
                 how_many_neighbours=NEIGHBOURS, collision_cube_min=CUBE_MIN)
        if kind == "hybrid":
            p.update(collision_type=api.COLLISION_FRAGMENTATION, N_tilde=4, pq_min_max=(C.c_int * 4)(0, 1, 0, 1),
                     mesh_brute_gravity=1)
        if "j2" in case.get("central", ""):
            p.update(J2_bool=1, J2=0.0, sideral_omega=2.0 * np.pi / 25.0)
        if "tides" in case.get("central", ""):
            p.update(central_tides_bool=1, k2=1.5, Delta_t=1e-3, dimensionless_moi=0.3307)
    return api.default_params(**p)


def _cells(n):
    return 1024 if n >= 500000 else 512 if n >= 100000 else 256


_engine = [None]  # what the library holds: slots and parameters of the last ncgpu_init


def _init(case):
    """ncgpu_init for the case, once for all the states that use it."""
    p = _params(case)
    n_max = 2 * case["n"] if case["kind"] == "hybrid" else case["n"] + case["n"] // 20 + 16
    key = (n_max, bytes(p))
    if _engine[0] != key:
        api.init(n_max, p)
        _engine[0] = key
    return n_max


def _pinned(a):
    """`a` in page-locked memory, as a host that steps on the device keeps its arrays."""
    t = torch.empty(a.shape, dtype=torch.from_numpy(a[:0]).dtype, pin_memory=True)
    v = t.numpy()
    v[...] = a
    return v


def _gamma(n, cells):
    return api.initial_gamma(n, cells, 0.5, 2.0, 0.015, NEIGHBOURS, CUBE_MIN)


def prepare(case, seed):
    n_max = _init(case)
    n, kind = case["n"], case["kind"]
    b, ex = _bodies(case, seed), _exists(case, seed)
    st = dict(kind=kind, case=case, cm=np.array(CENTRAL))
    if kind == "field":
        st["mode"] = api.GRAVITY_MODES[case["mode"]]
        if case["host"]:
            st.update(records=_pinned(b), ex=_pinned(ex), cm_acc=np.zeros(3))
        else:
            st.update(b=torch.from_numpy(b).cuda(), ex=torch.from_numpy(ex).cuda(),
                      acc=torch.zeros((n, 3), dtype=torch.float64, device="cuda"),
                      cm_acc=torch.zeros(3, dtype=torch.float64, device="cuda"))
            torch.cuda.synchronize()
    elif kind in ("adjoint", "forward"):
        st.update(args=(b[:, :3].copy(), b[:, 3:6].copy(), b[:, 6].copy(), b[:, 7].copy(), st["cm"], 1e-3, case["steps"]),
                  adj=np.random.default_rng([seed, 2]).normal(size=(n, 3)))
    elif kind == "output":
        cap = api.load().ncgpu_format_cartesian_cap()
        st.update(b=_pinned(b), ex=_pinned(ex), cap=cap, text=_pinned(np.zeros(cap, np.uint8)), end=0)
    else:
        st.update(b=_pinned(b), ex=_pinned(ex), b_out=_pinned(np.zeros((n_max, 8))), ex_out=_pinned(np.zeros(n_max, np.int32)),
                  lid=C.c_int(0), cm_out=np.zeros(8))
    return st


# --------------------------------------------------------------------- run --

def run(st):
    return {"field": _run_field, "bf": _run_bf, "mesh": _run_mesh, "hybrid": _run_hybrid, "output": _run_output,
            "forward": _run_forward, "adjoint": _run_adjoint}[st["kind"]](st)


def _run_field(st):
    lib, n = api.load(), st["case"]["n"]
    if st["case"]["host"]:  # the call leaves the accelerations in the records' velocity fields
        api.check(lib.ncgpu_vector_field(api.ptr(st["records"]), api.ptr(st["ex"]), n - 1, api.ptr(st["cm"]),
                                         api.ptr(st["cm_acc"]), st["mode"]), "ncgpu_vector_field")
        return st["records"][:, 3:6] * (st["ex"] != 0)[:, None], st["cm_acc"].copy()
    api.check(lib.ncgpu_vector_field_dev(C.c_void_p(st["b"].data_ptr()), C.c_void_p(st["ex"].data_ptr()), n - 1,
                                         api.ptr(st["cm"]), C.c_void_p(st["acc"].data_ptr()),
                                         C.c_void_p(st["cm_acc"].data_ptr()), st["mode"], None),
              "ncgpu_vector_field_dev")  # on the library's stream: its calls share one scratch
    return st["acc"], st["cm_acc"]


def _upload(st):
    api.upload(st["b"], st["ex"], st["cm"])


def _download(st):
    api.check(api.load().ncgpu_download(api.ptr(st["b_out"]), api.ptr(st["ex_out"]), C.byref(st["lid"]), api.ptr(st["cm_out"])),
              "ncgpu_download")
    k = st["lid"].value + 1
    return st["b_out"][:k], st["ex_out"][:k], st["cm_out"]


def _run_bf(st):
    _upload(st)
    api.set_timestep(1e-3)
    for _ in range(st["case"]["steps"]):
        hm = api.step_brute_force()
    return _download(st) + (hm,)


def _run_mesh(st):
    n, cells, dt = st["case"]["n"], _cells(st["case"]["n"]), 5e-4
    if "tides" in st["case"]["central"]:
        api.set_sideral_omega(2.0 * np.pi / 25.0)  # the tides of the last run have changed it
    _upload(st)
    gam = _gamma(n, cells)
    api.set_timestep(dt / 2)  # the half kick that integration_mesh starts with
    api.three_largest()
    _, _, tn = api.mesh(gam, False)
    api.kick()
    api.mesh_reset()
    api.set_timestep(dt)
    gam = api.update_gamma(gam, tn, n, NEIGHBOURS, CUBE_MIN / cells)
    for _ in range(st["case"]["steps"]):
        hm, tn = api.step_mesh(gam)
        gam = api.update_gamma(gam, tn, hm, NEIGHBOURS, CUBE_MIN / cells)
    return _download(st) + (hm, tn)


def _run_hybrid(st):
    cells = _cells(st["case"]["n"])
    _upload(st)
    api.set_timestep(2e-4)
    gam = CUBE_MIN / cells
    for _ in range(st["case"]["steps"]):
        hm, tn = api.step_mesh(gam)
        gam = api.update_gamma(gam, tn, hm, NEIGHBOURS, CUBE_MIN / cells)
    return _download(st) + (hm, tn)


def _run_output(st):
    _upload(st)
    api.snapshot_begin()
    lens = (C.c_ulong * 8)()
    api.check(api.load().ncgpu_format_cartesian(api.ptr(st["text"]), st["cap"], lens), "ncgpu_format_cartesian")
    stats, idx, cm, two = api.output_stats()
    api.snapshot_end()
    end = sum(lens)
    st["text"][end:st["end"]] = 0  # what a longer text before it left
    st["end"] = end
    return st["text"], np.array(lens[:], np.int64), stats, idx, cm, two


def _run_forward(st):
    return api.leapfrog(*st["args"])


def _run_adjoint(st):
    xf, vf = api.leapfrog(*st["args"])
    return (xf, vf) + api.leapfrog_vjp(*st["args"], st["adj"])


# -------------------------------------------------------------------- work --

def work(case):
    """Pair terms at 20 operations a force, 45 a vector-Jacobian product; each input read once, each output written once."""
    n, kind = case["n"], case["kind"]
    steps = case.get("steps", 1)
    if kind == "field":
        m = n * (1.0 - case["holes"])
        return {"bytes": 92.0 * n, "flops": 20.0 * m * m}
    if kind == "bf":  # and 20 operations of the collision predicate for each pair once
        return {"bytes": 136.0 * n, "flops": steps * 30.0 * n * n}
    if kind in ("mesh", "hybrid"):  # a state in and out, and a step's 208 bytes a body and 24 a pair (8 pairs a body)
        f = steps * (20.0 * n * n if kind == "hybrid" else 8.0 * n * 60.0)
        return {"bytes": (136.0 + steps * 400.0) * n, "flops": f}
    if kind == "output":  # records in, eight values of about 17 characters a body out
        return {"bytes": (68.0 + 8.0 * 17.0) * n, "flops": 8.0 * n}
    if kind == "forward":
        return {"bytes": 112.0 * n, "flops": 20.0 * steps * n * n}
    return {"bytes": 280.0 * n, "flops": (3 * 20.0 + 45.0) * steps * n * n}


# ------------------------------------------------------------------- exact --

def _pull(x, xj, eps):
    """Offsets from x's rows to xj's and their softened inverse distances cubed (0 where both are the same body)."""
    d = [xj[None, :, c] - x[:, None, c] for c in range(3)]
    r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
    same = r2 == 0.0
    r2 = r2 + eps * eps if eps is not None else r2
    r2 = torch.where(same, torch.ones_like(r2), r2)
    return d, torch.where(same, torch.zeros_like(r2), r2 ** -1.5)


def _field64(x, m, R, sp, X=None, rows=None):
    """Accelerations of the bodies (mutual and central mass 1 at X) and of the central body, in 64 bits."""
    n = x.shape[0]
    X = torch.zeros(3, dtype=x.dtype, device=x.device) if X is None else X
    rows = rows or max(1, min(n, (1 << 26) // n))
    out = []
    for lo in range(0, n, rows):
        hi = min(n, lo + rows)
        d, i3 = _pull(x[lo:hi], x, sp * (R[lo:hi, None] + R[None, :]) if sp else None)
        w = i3 * m[None, :]
        out.append(torch.stack([(w * d[c]).sum(1) for c in range(3)], 1))
    s = x - X
    c3 = (s * s).sum(1) ** -1.5
    return torch.cat(out) - s * c3[:, None], (m[:, None] * s * c3[:, None]).sum(0)


def _field64_vjp(x, m, R, sp, X, la, LA):
    """The field's vector-Jacobian product: gradients of sum(la . a) + LA . A in x, X and m."""
    n = x.shape[0]
    rows = max(1, min(n, (1 << 23) // n))
    x, m, X = (t.detach().requires_grad_() for t in (x, m, X))
    got = [torch.zeros_like(x), torch.zeros_like(m), torch.zeros_like(X)]
    for lo in range(0, n, rows):
        hi = min(n, lo + rows)
        d, i3 = _pull(x[lo:hi], x, sp * (R[lo:hi, None] + R[None, :]))
        w = i3 * m[None, :] * (la[lo:hi, 0, None] * d[0] + la[lo:hi, 1, None] * d[1] + la[lo:hi, 2, None] * d[2])
        for g, v in zip(got, torch.autograd.grad(w.sum(), (x, m, X), allow_unused=True)):
            if v is not None:
                g += v
    s = x - X
    c3 = (s * s).sum(1) ** -1.5
    v = (m[:, None] * s * c3[:, None]).sum(0) @ LA - (la * s * c3[:, None]).sum()
    for g, u in zip(got, torch.autograd.grad(v, (x, m, X))):
        g += u
    return got


def _exact_leapfrog(case, seed):
    st_b = torch.from_numpy(_bodies(case, seed)).cuda()
    x, v, m, R = st_b[:, :3].clone(), st_b[:, 3:6].clone(), st_b[:, 6].clone(), st_b[:, 7].clone()
    X, V = torch.zeros(3, dtype=x.dtype, device=x.device), torch.zeros(3, dtype=x.dtype, device=x.device)
    dt, seen = 1e-3, []
    x = x + dt / 2 * v
    for _ in range(case["steps"]):
        seen.append((x, X))
        a, A = _field64(x, m, R, SOFTENING, X)
        v, V = v + dt * a, V + dt * A
        x, X = x + dt * v, X + dt * V
    out = [x - dt / 2 * v, v]
    if case["kind"] == "forward":
        return tuple(t.cpu() for t in out)
    lx = torch.from_numpy(np.random.default_rng([seed, 2]).normal(size=(case["n"], 3))).cuda()
    lv, gm = -dt / 2 * lx, torch.zeros_like(m)
    LX, LV = torch.zeros_like(X), torch.zeros_like(V)
    for x, X in reversed(seen):
        lv, LV = lv + dt * lx, LV + dt * LX
        gx, g, GX = _field64_vjp(x, m, R, SOFTENING, X, lv, LV)
        lx, LX, gm = lx + dt * gx, LX + dt * GX, gm + dt * g
    return tuple(t.cpu() for t in out + [lx, lv + dt / 2 * lx, gm])


def exact(case, seed):
    """The fields and the leapfrog in 64 bits.  The stepping cases' states follow from collisions resolved one after
    another in the engine's order, and an output is text: those have no such value."""
    if case["kind"] in ("adjoint", "forward"):
        return _exact_leapfrog(case, seed)
    if case["kind"] != "field":
        return None
    ex = torch.from_numpy(_exists(case, seed)).cuda() != 0
    b = torch.from_numpy(_bodies(case, seed)).cuda()
    a, A = _field64(b[ex, :3], b[ex, 6], b[ex, 7], SOFTENING if case["soft"] else 0.0)
    acc = torch.zeros((case["n"], 3), dtype=torch.float64, device="cuda")
    acc[ex] = a
    return acc.cpu(), A.cpu()
