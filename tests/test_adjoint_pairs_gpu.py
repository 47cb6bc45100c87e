"""GPU: the differentiable leapfrog's pair sums at the edges of their tiling
(128-body tiles; blocks of one tile up to 16,384 bodies, of two beyond).

Small counts against torch's autograd of the same integrator in FP64 on the CPU;
past the change of block size through <w, J d> = <J^T w, d> with the JVP, whose
sums run body by body.  Tolerances, relative in the 2-norm:
  fp64   sums of at most ~700 additions in a row and terms of ~20 operations,
         1e-13 of the terms' absolute sum; a cancellation of 100 is allowed: 1e-11;
  mixed  a far term of the VJP moves by up to 5 (4.3 + 3.3) 6e-8 = 2.3e-6 (tile
         coordinates) + 5 x 1.2e-7 (reciprocal square root), FP32 runs of at most 32
         terms 1.9e-6; a cancellation of 4 is allowed: 2e-5.
"""
import numpy as np
import pytest
import torch

from conftest import make_params

pytestmark = pytest.mark.gpu
DT, STEPS = 0.02, 3


def bodies(n, radii, seed):
    from ncorpion_b200 import disks
    rng = np.random.default_rng(seed)
    b = disks.gravity_disk(n, seed=seed, radius=1e-2)
    b[:, 6] *= 3e5 / n  # the mutual pulls are of the central body's order
    if radii == "law":
        b[:, 7] = rng.uniform(5e-3, 5e-2, n)
    return b, rng


def final_x(x, v, m, R, sp):
    X, V = torch.zeros(3, dtype=x.dtype), torch.zeros(3, dtype=x.dtype)
    x, X = x + DT / 2 * v, X + DT / 2 * V
    eye = torch.eye(len(m), dtype=torch.bool)
    for _ in range(STEPS):
        d = x[None] - x[:, None]
        r2 = (d * d).sum(2) + (sp * (R[:, None] + R[None])) ** 2
        w = torch.where(eye, torch.zeros_like(r2), m[None] * torch.where(eye, torch.ones_like(r2), r2) ** -1.5)
        s = x - X
        c3 = (s * s).sum(1) ** -1.5
        a = (w[:, :, None] * d).sum(1) - s * c3[:, None]
        A = (m[:, None] * s * c3[:, None]).sum(0)
        v, V = v + DT * a, V + DT * A
        x, X = x + DT * v, X + DT * V
    return x - DT / 2 * v


@pytest.mark.parametrize("mode", [("exact", 1e-11), ("mixed", 2e-5)])
@pytest.mark.parametrize("radii", ["none", "equal", "law"])
@pytest.mark.parametrize("n", [1, 2, 33, 127, 128, 129, 257, 400])
def test_vjp_against_autograd(lib, n, radii, mode):
    from ncorpion_b200 import api
    b, rng = bodies(n, radii, n)
    sp = 0.0 if radii == "none" else 0.5
    api.init(n, make_params(softening_parameter=sp, gravity_mode=api.GRAVITY_MODES[mode[0]]))
    adj = rng.normal(size=(n, 3))
    cm = np.array([0, 0, 0, 0, 0, 0, 1.0, 1.0])
    args = (b[:, :3], b[:, 3:6], b[:, 6], b[:, 7], cm, DT, STEPS)
    xf, _ = api.leapfrog(*args, checkpoint=2)
    got = api.leapfrog_vjp(*args, adj, checkpoint=2)
    t = [torch.from_numpy(np.ascontiguousarray(q)).requires_grad_() for q in (b[:, :3], b[:, 3:6], b[:, 6])]
    x = final_x(*t, torch.from_numpy(b[:, 7].copy()), sp)
    ref = torch.autograd.grad((x * torch.from_numpy(adj)).sum(), t)
    assert np.linalg.norm(xf - x.detach().numpy()) <= mode[1] * np.linalg.norm(xf)
    for g, r in zip(got, ref):
        assert np.linalg.norm(g - r.numpy()) <= mode[1] * np.linalg.norm(r.numpy())
    again = api.leapfrog_vjp(*args, adj, checkpoint=2)
    assert all(np.array_equal(p, q) for p, q in zip(got, again))
    api.finalize()


@pytest.mark.parametrize("mode", ["exact", "mixed"])
def test_vjp_in_place(lib, mode):
    """x_final may be the array that brings dL/dx_final, the gradients those of the initial state."""
    import ctypes as C
    from ncorpion_b200 import api
    n = 300
    b, rng = bodies(n, "equal", 8)
    adj = rng.normal(size=(n, 3))
    cm = np.array([0, 0, 0, 0, 0, 0, 1.0, 1.0])
    api.init(n, make_params(softening_parameter=0.5, gravity_mode=api.GRAVITY_MODES[mode]))
    args = (b[:, :3], b[:, 3:6], b[:, 6], b[:, 7], cm, DT, STEPS)
    xf, _ = api.leapfrog(*args)
    ref = api.leapfrog_vjp(*args, adj)
    x, v, m, R, xa = (np.array(q, order="C") for q in (b[:, :3], b[:, 3:6], b[:, 6], b[:, 7], adj))
    p = [q.ctypes.data for q in (x, v, m, R, cm, xa)]
    a = api.LeapfrogArgs(n, *p[:5], DT, STEPS, 32, p[5], None, p[5], p[0], p[1], p[2])
    api.check(api.load().ncgpu_leapfrog_vjp(C.byref(a)), "ncgpu_leapfrog_vjp")
    for got, want in zip((xa, x, v, m), (xf, *ref)):
        assert np.array_equal(got, want)
    api.finalize()


@pytest.mark.parametrize("n", [16384, 16385, 16650])
def test_vjp_past_the_block_size(lib, n):
    from ncorpion_b200 import api
    b, rng = bodies(n, "equal", 5)
    b[:, 6] *= 1e-2
    adj = rng.normal(size=(n, 3))
    tan = (rng.normal(size=(n, 3)), rng.normal(size=(n, 3)), b[:, 6] * rng.normal(size=n))
    cm = np.array([0, 0, 0, 0, 0, 0, 1.0, 1.0])
    args = (b[:, :3], b[:, 3:6], b[:, 6], b[:, 7], cm, DT, 2)
    got = {}
    for mode in ("exact", "mixed"):
        api.init(n, make_params(softening_parameter=0.5, gravity_mode=api.GRAVITY_MODES[mode]))
        got[mode] = api.leapfrog_vjp(*args, adj)
        if mode == "exact":
            out = api.leapfrog_jvp(*args, *tan)
            lhs, rhs = float((adj * out).sum()), float(sum((g * d).sum() for g, d in zip(got[mode], tan)))
            assert abs(lhs - rhs) <= 1e-11 * np.linalg.norm(adj) * np.linalg.norm(out)
    for g, r in zip(got["mixed"], got["exact"]):
        assert np.linalg.norm(g - r) <= 2e-5 * np.linalg.norm(r)
    api.finalize()


@pytest.mark.parametrize("radii", ["none", "equal", "law"])
@pytest.mark.parametrize("mode", ["exact", "mixed"])
def test_units(lib, mode, radii):
    """Lengths times 2^k, masses times 2^j and G times 2^(3k - j): the positions times 2^k, the gradients
    to positions and velocities as they were, those to masses times 2^(k - j).  The powers of two
    pass through every operation but the FP64 reciprocal square root unchanged: the fp64 bound above."""
    from ncorpion_b200 import api
    n = 3000
    b, rng = bodies(n, radii, 4)
    sp = 0.0 if radii == "none" else 0.5
    adj = rng.normal(size=(n, 3))

    def run(k, j):
        L, W = 2.0 ** k, 2.0 ** j
        api.init(n, make_params(softening_parameter=sp, gravity_mode=api.GRAVITY_MODES[mode], G=2.0 ** (3 * k - j)))
        cm = np.array([0, 0, 0, 0, 0, 0, W, L])
        args = (b[:, :3] * L, b[:, 3:6] * L, b[:, 6] * W, b[:, 7] * L, cm, DT, STEPS)
        x, _ = api.leapfrog(*args)
        gx, gv, gm = api.leapfrog_vjp(*args, adj)
        api.finalize()
        return x / L, gx, gv, gm * (W / L)

    base = run(0, 0)
    for k, j in [(-60, -60), (-45, 40), (20, 60), (30, -30), (42, 0), (50, 60)]:
        for p, q in zip(run(k, j), base):
            assert np.linalg.norm(p - q) <= 1e-11 * np.linalg.norm(q), (k, j)
