"""With "fvx" asked for, the finite-volume elements of a mixed mesh are rounded in the
reference's order throughout, the traces of their DG neighbours included: on meshes whose
outer faces they do not touch the right-hand side equals the oracle's bit for bit."""
import numpy as np
import pytest

import nmesh_gb300 as ng
from helpers import RTOL_RHS, gaussian_pulses, oracle_for, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _gpu(cuda_ok):
    yield


@pytest.mark.parametrize("n,luni", [(2, 0), (3, 1), (5, 0), (6, 1), (7, 1), (9, 0), (12, 0)])
@pytest.mark.parametrize("flux", ["LLF", "upwind"])
def test_finite_volume_elements_equal_the_oracle(n, luni, flux):
    rec, extrap = ("WENOm5_2", "dnfn_extrap1") if n >= 5 else ("1", "no")
    m = ng.Mesh.build(ng.MESH_CUBEDSPHERES7, n=n, luni=luni, cs_dc=1.0, cs_r0fac=20.0, fv=[0])
    u = gaussian_pulses(m.coords(), seed=n, rmin=1.0, rmax=6.0)
    u += 1e-2 * np.random.default_rng(n).standard_normal(u.shape)
    ev = ng.Evolution(m, ng.BC_OUTGOING)
    ev.set_fv(rec, extrap)
    ev.set_numflux(flux)
    ev.set_kernel("eo")
    ev.set_kernel("fvx")
    r = ev.rhs(u, 0.0)
    want = oracle_for(m, bc=1, fv_rec=rec, fv_extrap=extrap, numflux=flux).rhs(u, 0.0)
    fv = m.fv() != 0
    assert fv.any() and (m.faces()[0][fv] >= 0).all()
    assert np.array_equal(r[fv], want[fv])
    assert rel_l2(r, want) <= RTOL_RHS
