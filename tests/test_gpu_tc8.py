"""The eight-digit kernel at n = 7 and 9 ("tc8"): the checks of the other kernels of
stage_tcs.cu, and where the autotuner takes it in the place of the seven-digit "tc"."""
import numpy as np
import pytest

import nmesh_gb300 as ng
import test_gpu_tcs
import test_gpu_tcs_lines
from helpers import PI

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _gpu(cuda_ok):
    yield


@pytest.mark.parametrize("n", [7, 9])
def test_like_the_other_orders(n):
    for numflux, method in (("LLF", "RK4"), ("upwind", "sspRK3")):
        test_gpu_tcs.test_shells_vs_oracle(n, "tc8", numflux, method)
    test_gpu_tcs.test_periodic_box_vs_oracle(n, "tc8")
    test_gpu_tcs.test_refined_mesh_and_element_lists(n, "tc8")
    test_gpu_tcs.test_mixed_mesh(n, "tc8")
    test_gpu_tcs.test_zeros_nan_and_dynamic_range(n, "tc8")
    for field, out in ((0, 1), (1, 0)):
        test_gpu_tcs_lines.test_every_line_has_its_own_scale(n, "tc8", field, out)
    test_gpu_tcs_lines.test_a_nan_spoils_its_lines_only(n, "tc8")
    test_gpu_tcs_lines.test_values_below_the_normal_range(n, "tc8")


def _candidates(info):
    return {s.split(":")[0] for s in info.split() if "=" in s}


@pytest.mark.parametrize("n,kind,digits", [(7, "box", 8), (7, "mixed", 8), (7, "shells", 7), (9, "box", 7),
                                           (9, "mixed", 7), (9, "shells", 7)])
def test_candidates_of_the_autotuner(n, kind, digits):
    if kind == "box":
        m = ng.Mesh.build(ng.MESH_BOX, n=n, luni=3, xc=(PI, PI, PI), box_dout=PI, periodic=True)
    else:
        m = ng.Mesh.build(ng.MESH_CUBEDSPHERES7, n=n, luni=2, cs_dc=1.0, cs_r0fac=20.0,
                          fv=[0, 2] if kind == "mixed" else False)
    ev = ng.Evolution(m, ng.BC_OUTGOING)
    ev.rhs(np.zeros((m.nelem, 5, m.np)))
    timed = _candidates(ev.kernel_info())
    assert ("tc8" in timed) == (digits == 8) and ("tc" in timed) == (digits == 7)
    ev.set_kernel("tc")
    ev.set_kernel("tc8")
    if kind == "mixed":
        ev.set_kernel("fvx:1:512")


@pytest.mark.parametrize("n", [7, 9])
def test_batches_keep_fp64_accuracy(n):
    """One step of a pulse that fills a small part of the elements' range: orders side by
    side and the persistent FP64 kernel agree to FP64 rounding on every line."""
    meshes = [ng.Mesh.build(ng.MESH_BOX, n=k, luni=3, xc=(PI, PI, PI), box_dout=PI, periodic=True)
              for k in (n, 5)]
    res = []
    for mode in (1, 2):
        b = ng.Batch(meshes, ng.BC_OUTGOING)
        b.set_mode(mode)
        rng = np.random.default_rng(n)
        for p, m in enumerate(meshes):
            u = np.zeros(b.shape(p))
            u[:, 0] = rng.standard_normal(u[:, 0].shape)
            # the lower half of every element's lines a millionth of the upper half's
            u[:, 0].reshape(m.nelem, m.n, -1)[:, : m.n // 2] *= 1e-9
            b.set_state(p, u)
        b.rk4_steps(0.0, 1e-12, 1)
        res.append(b.get_state(0)[:, 1])
    n2 = meshes[0].n ** 2
    # r_c_x dt on the small planes: 1e-12 x 1e-9 x O(n^2), within FP64 rounding of it
    small = [r.reshape(len(r), -1, n2)[:, 1:n // 2 - 1] for r in res]
    assert np.abs(small[0] - small[1]).max() <= 1e-13 * np.abs(small[0]).max()
