"""Lines of the digit-product kernels of stage_tcs.cu stand on their own, as those of the
FP64 kernels do: a line's derivative depends on no other line's size, a NaN spoils the lines
through it and no others, and values below the normal range count.

On a periodic box, with pi alone (c_x alone) not zero, r_c_x (r_pi) comes from the lines
along x and the jumps at their ends.  Data that are scaled by a power of two on each line give
the result scaled by it, bit for bit, as long as nothing leaves the normal range; a grid common
to the element's lines would lose the small ones' digits."""
import numpy as np
import pytest

import nmesh_gb300 as ng
from helpers import PI

pytestmark = pytest.mark.gpu

CASES = [(n, "tc") for n in (4, 5, 6, 8, 10)] + [(n, "tcl") for n in range(6, 11)]
VJP = [(n, "tcvjp") for n in (4, 5, 6, 10)] + [(n, "tcvjw") for n in (4, 5, 7, 8, 9, 10)]


@pytest.fixture(autouse=True)
def _gpu(cuda_ok):
    yield


def _box(n):
    return ng.Mesh.build(ng.MESH_BOX, n=n, luni=1, xc=(PI, PI, PI), box_dout=PI, periodic=True)


def _scaled(n, field):
    """Fields of order one and the same with every line along x times a power of two."""
    rng = np.random.default_rng(n + field)
    u = np.zeros((8, 5, n ** 3))
    u[:, field] = rng.standard_normal((8, n ** 3))
    amp = np.repeat(2.0 ** -rng.integers(0, 60, n * n), n)
    amp[:n] = 1.0
    return u, u * amp, amp


def _transposed(m, variant, x):
    import torch
    ev = ng.Evolution(m, ng.BC_OUTGOING)
    if variant:
        ev.set_kernel(variant)
    rbar, wbar = torch.as_tensor(x).cuda(), torch.empty(x.shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ev.rhs_vjp_device(rbar.data_ptr(), wbar.data_ptr())
    return wbar.cpu().numpy()


@pytest.mark.parametrize("field,out", [(0, 1), (1, 0)])
@pytest.mark.parametrize("n,variant", CASES + [(n, "eo") for n in (4, 9)])
def test_every_line_has_its_own_scale(n, variant, field, out):
    u, small, amp = _scaled(n, field)
    ev = ng.Evolution(_box(n), ng.BC_OUTGOING)
    ev.set_kernel(variant)
    want = ev.rhs(u)[:, out] * amp
    assert np.abs(want).min(axis=0).max() > 0
    assert np.array_equal(ev.rhs(small)[:, out], want)


@pytest.mark.parametrize("field,out", [(0, 1), (1, 0)])
@pytest.mark.parametrize("n,variant", VJP + [(4, "vjp"), (9, "vjp")])
def test_every_transposed_line_has_its_own_scale(n, variant, field, out):
    u, small, amp = _scaled(n, field)
    assert np.array_equal(_transposed(_box(n), variant, small)[:, out],
                          _transposed(_box(n), variant, u)[:, out] * amp)


@pytest.mark.parametrize("field,out", [(0, 1), (1, 0)])
@pytest.mark.parametrize("n", [7, 9])
def test_the_line_left_over_has_its_own_scale(n, field, out):
    """49 and 81 lines are 3 and 5 tiles and a line, which is an FP64 dot product ("tc" and
    "tcvjp" at n = 7 and 9; their tiles have one grid per element)."""
    u, _, _ = _scaled(n, field)
    small = u.copy()
    small[:, :, -n:] *= 2.0 ** -40
    ev = ng.Evolution(_box(n), ng.BC_OUTGOING)
    ev.set_kernel("tc")
    assert np.array_equal(ev.rhs(small)[:, out, -n:], ev.rhs(u)[:, out, -n:] * 2.0 ** -40)
    got, want = (_transposed(_box(n), "tcvjp", x)[:, out, -n:] for x in (small, u))
    assert np.array_equal(got, want * 2.0 ** -40)


@pytest.mark.parametrize("n,variant", CASES)
def test_a_nan_spoils_its_lines_only(n, variant):
    rng = np.random.default_rng(n)
    m = ng.Mesh.build(ng.MESH_CUBEDSPHERES7, n=n, luni=0, cs_dc=1.0, cs_r0fac=20.0)
    u = rng.standard_normal((m.nelem, 5, m.np))
    mid = 1 + n + n * n  # an interior node
    u[0, 0, mid] = u[3, 2, mid] = np.nan
    bad = []
    for k in ("eo", variant):
        ev = ng.Evolution(m, ng.BC_OUTGOING)
        ev.set_kernel(k)
        bad.append(np.isnan(ev.rhs(u)))
    assert bad[0].any() and np.array_equal(bad[0], bad[1])


@pytest.mark.parametrize("n,variant", CASES)
def test_values_below_the_normal_range(n, variant):
    """Whole multiples of the smallest number: either kernel rounds each of its sums of up
    to n products, the chain rule's and the lift's to a multiple of it."""
    rng = np.random.default_rng(n)
    u = rng.integers(-1000, 1000, (8, 5, n ** 3)) * 2.0 ** -1074
    r = []
    for k in ("eo", variant):
        ev = ng.Evolution(_box(n), ng.BC_OUTGOING)
        ev.set_kernel(k)
        r.append(ev.rhs(u))
    assert np.abs(r[0]).max() > 1000 * 2.0 ** -1074
    # three directions of n products, six faces of four terms
    assert np.abs(r[0] - r[1]).max() / 2.0 ** -1074 <= 3 * (n + 2) + 24


@pytest.mark.parametrize("n,few,many", [(6, "vjp", "tcvjp"), (7, "tcvjw", "tcvjp"), (9, "tcvjw", "tcvjp"),
                                        (11, "vjp", "vjp")])
def test_choice_of_the_transposed_kernel(n, few, many):
    """By the number of SMs: 64 elements have room at once, 4096 have not (the kernels differ
    in their last bits)."""
    for luni, name in ((2, few), (4, many)):
        m = ng.Mesh.build(ng.MESH_BOX, n=n, luni=luni, xc=(PI, PI, PI), box_dout=PI, periodic=True)
        x = np.random.default_rng(n).standard_normal((m.nelem, 5, m.np))
        got = _transposed(m, None, x)
        for k in {"vjp", few, many}:
            assert np.array_equal(got, _transposed(m, k, x)) == (k == name), (luni, k)
