"""The finite-volume scratch ("fvc") of a context that can switch elements is sized for the
elements that are finite volume, and grows with them; the results are those of a context made
with them."""
import numpy as np
import pytest

import nmesh_gb300 as ng

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _gpu(cuda_ok):
    yield


def test_scratch_grows_with_the_finite_volume_elements():
    import torch
    n = 9
    m = ng.Mesh.build(ng.MESH_CUBEDSPHERES7, n=n, luni=2, cs_dc=1.0, cs_r0fac=20.0)
    u = np.random.default_rng(1).standard_normal((m.nelem, 5, m.np))
    ev = ng.Evolution(m, ng.BC_OUTGOING, switchable=True)
    ev.set_fv("WENOm5_2", "dnfn_extrap1")
    ev.set_kernel("eo")
    ev.set_kernel("fvc")
    ev.rhs(u)
    few = np.zeros(m.nelem, np.int32)
    few[:4] = 1
    ev.set_element_types(few)
    ev.rhs(u)
    free = torch.cuda.mem_get_info()[0]
    half = np.zeros(m.nelem, np.int32)
    half[: m.nelem // 2] = 1
    ev.set_element_types(half)
    scratch = 12 * 8 * n ** 3 * (m.nelem // 2)
    assert free - torch.cuda.mem_get_info()[0] >= 0.8 * scratch
    ref = ng.Evolution(ng.Mesh.build(ng.MESH_CUBEDSPHERES7, n=n, luni=2, cs_dc=1.0, cs_r0fac=20.0),
                       ng.BC_OUTGOING, switchable=True)
    ref.set_element_types(half)
    ref.set_fv("WENOm5_2", "dnfn_extrap1")
    ref.set_kernel("eo")
    ref.set_kernel("fvc")
    assert np.array_equal(ev.rhs(u), ref.rhs(u))
