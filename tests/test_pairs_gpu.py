"""GPU: the tiled gravity's pair sums (every unordered pair once) at the sizes
where their tiling changes: remainders of 128-body tiles, one tile, an odd and
an even number of blocks, the block sizes' limits and a body count whose partial
rows are summed in several shares.

Errors are taken relative to the sum of the absolute values of a body's terms
(numpy, FP64, on a sample of bodies), so that cancellation plays no part.
  fp64   a sum is at most ~700 additions in a row (512 of a block's columns, the
         blocks' rows): 700 x 1.1e-16 = 7.7e-14, the terms ~1e-15: 1e-13.
  mixed  far tiles are at least 0.15 box diagonals apart, so a coordinate
         relative to the tile's centre is at most ~4.3 distances and its FP32
         rounding moves a term by up to 3 (4.3 + 3.3) 6e-8 = 1.4e-6; runs of 32
         FP32 additions 1.9e-6; the reciprocal square root 3 x 1.2e-7: 4e-6.
"""
import numpy as np
import pytest

from conftest import make_params

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 33, 127, 128, 129, 256, 257, 385, 1000, 12288, 12289, 16384, 16385, 16641, 65408, 65537, 160001,
         12290, 16386, 49024, 49026]  # (the odd ones have empty slots; blocks of 1, 2, 2 and 4 tiles)


def reference(b, ex, sp, rows):
    """Accelerations of the bodies `rows` and the sums of their terms' absolute values."""
    on = ex != 0
    acc, mag = np.zeros((len(rows), 3)), np.zeros((len(rows), 3))
    for q, k in enumerate(rows):
        d = b[on, :3] - b[k, :3]
        r2 = (d * d).sum(1) + (sp * (b[k, 7] + b[on, 7])) ** 2
        self_ = np.flatnonzero(on) == k
        r2[self_] = 1.0
        t = (b[on, 6] * np.where(self_, 0.0, r2 ** -1.5))[:, None] * d
        acc[q], mag[q] = t.sum(0), np.abs(t).sum(0)
    return acc, mag


@pytest.mark.parametrize("radii", ["none", "equal", "law"])
@pytest.mark.parametrize("n", SIZES)
def test_pair_sums(lib, n, radii):
    from ncorpion_b200 import api, disks
    if n > 70000 and radii == "law":
        pytest.skip("the several-share sums do not depend on the softening")
    b = disks.gravity_disk(n, seed=n)
    rng = np.random.default_rng(n)
    if radii == "law":
        b[:, 7] = disks.powerlaw_radii(rng, n, 1e-5, 1e-3)
    ex = np.ones(n, np.int32)
    if n % 2:
        ex[rng.random(n) < 0.04] = 0
        ex[0] = 1
    sp = 0.0 if radii == "none" else 0.5
    api.init(n, make_params(softening_parameter=sp, central_mass_bool=0))
    live = np.flatnonzero(ex)
    rows = live if len(live) <= 48 else np.sort(rng.choice(live, 48, replace=False))
    ref, mag = reference(b, ex, sp, rows)
    scale = mag.max(axis=1, keepdims=True) + 1e-300
    for mode, tol in (("fp64", 1e-13), ("mixed", 4e-6)):
        acc, _ = api.vector_field(b, ex, mode=mode)
        assert np.all(np.isfinite(acc)) and not acc[ex == 0].any()
        err = np.abs(acc[rows] - ref) / scale
        assert err.max() <= tol, (mode, err.max())
        again, _ = api.vector_field(b, ex, mode=mode)
        assert np.array_equal(acc, again)  # the sums' order is fixed
    api.finalize()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 4095, 4097, 14336, 14337])
def test_equal_keys(lib, n):
    """Bodies at 64 places, so that nearly all Morton keys have equals (a stable
    order places each once), with holes; the same bounds as above."""
    from ncorpion_b200 import api, disks
    b = disks.gravity_disk(n, seed=n)
    rng = np.random.default_rng(n)
    b[:, :3] = b[rng.integers(0, min(n, 64), n), :3]
    ex = np.ones(n, np.int32)
    ex[rng.random(n) < 0.1] = 0
    ex[n - 1] = 1
    api.init(n, make_params(softening_parameter=0.5, central_mass_bool=0))
    live = np.flatnonzero(ex)
    rows = live if len(live) <= 48 else np.sort(rng.choice(live, 48, replace=False))
    ref, mag = reference(b, ex, 0.5, rows)
    scale = mag.max(axis=1, keepdims=True) + 1e-300
    for mode, tol in (("fp64", 1e-13), ("mixed", 4e-6)):
        acc, _ = api.vector_field(b, ex, mode=mode)
        assert np.all(np.isfinite(acc)) and not acc[ex == 0].any()
        assert (np.abs(acc[rows] - ref) / scale).max() <= tol
    api.finalize()


@pytest.mark.parametrize("radii", ["none", "equal", "law"])
@pytest.mark.parametrize("n", [3000, 17000])
def test_units(lib, n, radii):
    """The caller's units are not bound to FP32's range: lengths times 2^k and masses times 2^j
    (0.3 astronomical units are 2^42 cm) give the accelerations times 2^(j - 2k).  The powers of two pass
    through every operation but the FP64 reciprocal square root unchanged: the fp64 bound above."""
    from ncorpion_b200 import api, disks
    b = disks.gravity_disk(n, seed=n)
    rng = np.random.default_rng(n)
    b[:, 7] = disks.powerlaw_radii(rng, n, 1e-5, 1e-3) if radii == "law" else 1e-3
    ex = np.ones(n, np.int32)
    sp = 0.0 if radii == "none" else 0.5
    api.init(n, make_params(softening_parameter=sp, central_mass_bool=0))
    rows = np.arange(0, n, n // 40)
    _, mag = reference(b, ex, sp, rows)
    scale = mag.max(axis=1, keepdims=True)
    for mode in ("fp64", "mixed"):
        base, _ = api.vector_field(b, ex, mode=mode)
        for k, j in [(-60, -60), (-45, 40), (0, -60), (20, 60), (42, 0), (44, -30), (50, 60)]:
            u = b.copy()
            u[:, [0, 1, 2, 7]] *= 2.0 ** k
            u[:, 6] *= 2.0 ** j
            acc, _ = api.vector_field(u, ex, mode=mode)
            err = np.abs(acc * 2.0 ** (2 * k - j) - base)[rows] / scale
            assert err.max() <= 1e-13, (mode, k, j, err.max())
    api.finalize()


def test_short_of_memory(lib):
    """With 160 MB left on the device the partial rows (1 GB here for the field, 0.4 GB for the leapfrog's VJP)
    are summed in more and smaller shares, grouped differently: the fp64 bound above."""
    import torch
    from ncorpion_b200 import api, disks
    n, m = 160001, 60000
    b = disks.gravity_disk(n, seed=1)
    p = make_params(softening_parameter=0.5, central_mass_bool=0, gravity_mode=api.GRAVITY_MIXED)
    cm = np.array([0, 0, 0, 0, 0, 0, 1.0, 1.0])
    args = (b[:m, :3], b[:m, 3:6], b[:m, 6], b[:m, 7], cm, 1e-3, 1, np.ones((m, 3)))

    def run():
        grads = api.leapfrog_vjp(*args)
        return [*grads, api.vector_field(b, mode="mixed")[0]]

    api.init(n, p)
    full = run()
    api.finalize()
    api.init(n, p)
    api.vector_field(b[:256], mode="mixed")
    torch.cuda.synchronize()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (160 << 20), dtype=torch.uint8, device="cuda")
    try:
        short = run()
    finally:
        del hog
        torch.cuda.empty_cache()
        api.finalize()
    for s, f in zip(short, full):
        assert np.linalg.norm(s - f) <= 1e-13 * np.linalg.norm(f)
