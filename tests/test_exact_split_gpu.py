"""GPU: the exact force kernel at the edges of its split (8 targets a CTA, rounds
of 64 sources, 256 bodies a round of CM_acc, one preparation CTA up to 8,192 slots,
512 threads a CTA up to 2,048): bit-identical to the oracle, with empty slots, with
softening and J2 on and off, with bodies whose offsets are signed zeros, and in parts."""
import numpy as np
import pytest

from conftest import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("soft,j2", [(0.0, 0), (0.5, 1)])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 63, 64, 65, 255, 257, 513, 2047, 2049, 2600])
def test_bits(lib, port, n, soft, j2):
    from ncorpion_b200 import api, disks
    rng = np.random.default_rng(n)
    b = disks.gravity_disk(n, seed=n)
    if n >= 63:  # planes of equal coordinates, of either sign of zero
        b[: n // 3, 2] = 0.0
        b[n // 4: n // 3, 2] = -0.0
        b[5:20, 0] = b[5, 0]
    ex = np.ones(n, np.int32)
    if n > 8:
        ex[rng.random(n) < 0.1] = 0
    cm = np.array([1e-6, -2e-6, 0.0, 0, 0, 0, 1.0, 1.0])
    p = make_params(softening_parameter=soft, J2_bool=j2, J2=1e-3 if j2 else 0.0)
    api.init(n, p)
    ref, cref = port.vector_field(b, ex, cm, p)
    acc, cma = api.vector_field(b, ex, cm, mode="exact")
    assert np.array_equal(acc.view(np.int64)[ex == 1], np.ascontiguousarray(ref).view(np.int64)[ex == 1])
    assert np.array_equal(cma, cref)
    api.finalize()


@pytest.mark.parametrize("nparts", [2, 3, 7])
@pytest.mark.parametrize("n", [7, 9, 65, 2049])
def test_bits_in_parts(lib, n, nparts):
    """Parts that end inside a CTA's 8 targets, and parts without a target: each row from one part (-0.0
    from the others), their sum and every part's CM_acc bit for bit the whole's."""
    import ctypes as C
    import torch
    from ncorpion_b200 import api, disks
    ex = np.ones(n, np.int32)
    ex[::5] = 0
    cm = np.array([1e-6, -2e-6, 0.0, 0, 0, 0, 1.0, 1.0])
    d_b, d_ex = torch.from_numpy(disks.gravity_disk(n, seed=n)).cuda(), torch.from_numpy(ex).cuda()
    api.init(n, make_params(softening_parameter=0.5))

    def run(part, parts):
        acc, cma = (torch.full(s, np.nan, dtype=torch.float64, device="cuda") for s in ((n, 3), (3,)))
        api.check(lib.ncgpu_vector_field_part(*(C.c_void_p(t.data_ptr()) for t in (d_b, d_ex)), n - 1, api.ptr(cm), part,
                                              parts, *(C.c_void_p(t.data_ptr()) for t in (acc, cma)), 0, None), "part")
        torch.cuda.synchronize()
        return acc.cpu().numpy(), cma.cpu().numpy()

    full, cma = run(0, 1)
    total, owners = np.full_like(full, -0.0), np.zeros(n, int)
    for part in range(nparts):
        acc, c = run(part, nparts)
        assert np.array_equal(c, cma)
        owners += ~(acc.view(np.int64) == np.float64(-0.0).view(np.int64)).all(axis=1)
        total = total + acc
    assert np.array_equal(total.view(np.int64), full.view(np.int64)) and (owners[ex == 1] == 1).all()
    api.finalize()


def test_past_the_preparation_cta(lib, port):
    """8,192 and 8,193 slots with most of them empty: the two compactions give the same field."""
    from ncorpion_b200 import api, disks
    p = make_params(softening_parameter=0.5)
    cm = np.array([0.0, 0, 0, 0, 0, 0, 1.0, 1.0])
    b = disks.gravity_disk(8193, seed=1)
    ex = (np.random.default_rng(0).random(8193) < 0.1).astype(np.int32)
    ex[8192] = 0
    api.init(8193, p)
    ref, cref = port.vector_field(b, ex, cm, p)
    for k in (8192, 8193):
        acc, cma = api.vector_field(b[:k], ex[:k], cm, mode="exact")
        assert np.array_equal(acc, ref[:k] * (ex[:k] != 0)[:, None]) and np.array_equal(cma, cref)
    api.finalize()


def test_no_slots_leave_the_kernel_time(lib):
    """A field of no slots runs no field kernel: no time before the first one, that one's after it."""
    from ncorpion_b200 import api, disks
    none = np.zeros((0, 8))
    api.init(64, make_params())
    for mode in ("exact", "fp64", "mixed"):
        api.vector_field(none, mode=mode)
        with pytest.raises(api.NcgpuError) as e:
            api.last_kernel_ms()
        assert e.value.status == api.E_STATE
    api.vector_field(disks.gravity_disk(64, seed=1))
    t = api.last_kernel_ms()
    for mode in ("exact", "fp64", "mixed"):
        api.vector_field(none, mode=mode)
        assert api.last_kernel_ms() == t
    api.finalize()


@pytest.mark.parametrize("n", [8192, 8193])
def test_unknown_mode(lib, n):
    """A mode that is none of the three: the exact field up to 8,192 slots, refused beyond when a slot is filled."""
    from ncorpion_b200 import api, disks
    b, ex = disks.gravity_disk(n, seed=2), np.zeros(n, np.int32)
    api.init(n, make_params())
    for live in (0, 5):
        ex[:live] = 1
        if live and n > 8192:
            with pytest.raises(api.NcgpuError) as e:
                api.vector_field(b, ex, mode=7)
            assert e.value.status == api.E_ARG
        else:
            got, ref = api.vector_field(b, ex, mode=7), api.vector_field(b, ex, mode="exact")
            assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    api.finalize()
