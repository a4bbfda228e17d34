"""The streamed host round trip in several chunks (rk4_steps_host): chunks of the last
stage alternate between two streams while results are copied back, and a single step of a
conforming DG mesh also starts its first stage by element lists as the copy in proceeds.
Every element sees the arithmetic of a resident step, so the results are equal bit for
bit.  NMG_COPY_CHUNKS sets the number of chunks of the contexts made after it; without it
a mesh of at least 896 elements and 10 MB has more than one."""
import numpy as np
import pytest

import nmesh_gb300 as ng
from helpers import PI

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _gpu(cuda_ok):
    yield


def _mesh(kind, n, luni, **kw):
    if kind == "box":
        return ng.Mesh.build(ng.MESH_BOX, n=n, luni=luni, xc=(PI, PI, PI), box_dout=PI, periodic=True, **kw)
    return ng.Mesh.build(ng.MESH_CUBEDSPHERES7, n=n, luni=luni, cs_dc=1.0, cs_r0fac=20.0, **kw)


def _equal(m, variant, dt, steps, repeats=1):
    u = np.random.default_rng(m.n).standard_normal((m.nelem, 5, m.np))
    ev = ng.Evolution(m, ng.BC_OUTGOING)
    if variant:
        ev.set_kernel(variant)
    ev.set_state(u)
    ev.rk4_steps(0.0, dt, steps)
    want = ev.get_state()
    for _ in range(repeats):
        assert np.array_equal(ev.rk4_steps_host(u, 0.0, dt, steps), want)
    ev.close()


@pytest.mark.parametrize("chunks", [2, 8, 16, 32])
@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("kind,n,luni", [("box", 6, 2), ("shells", 9, 1), ("shells", 4, 2), ("box", 13, 1)])
def test_finite_volume_mesh(monkeypatch, kind, n, luni, steps, chunks):
    """The two streams' scratch halves; 32 chunks of the 8-element box are single elements."""
    monkeypatch.setenv("NMG_COPY_CHUNKS", str(chunks))
    _equal(_mesh(kind, n, luni, fv=True), "", 1e-3, steps, repeats=3)


@pytest.mark.parametrize("steps", [1, 3])
def test_finite_volume_mesh_by_size(steps):
    """3584 elements of 7^3 points: eight chunks by the size rule."""
    _equal(_mesh("shells", 7, 3, fv=True), "", 1e-3, steps, repeats=3)


@pytest.mark.parametrize("variant,kernels", [("fvc", 2), ("fvx", 1), ("fv", 1)])
def test_launches_of_a_chunked_finite_volume_step(monkeypatch, variant, kernels):
    """Every kernel counts: a chunk of "fvc" is two launches."""
    monkeypatch.setenv("NMG_COPY_CHUNKS", "8")
    m = _mesh("box", 5, 2, fv=True)
    ev = ng.Evolution(m, ng.BC_OUTGOING)
    ev.set_kernel(variant)
    u = np.zeros((m.nelem, 5, m.np))
    before = ev.launches
    ev.rk4_steps_host(u, 0.0, 1e-3, 1)
    assert ev.launches - before == (3 + 8) * kernels
    ev.close()


DG = [(n, "tc") for n in range(4, 11)] + [(8, "tc:1:256"), (10, "tc:1:256")]
DG += [(n, "tcl") for n in range(6, 11)] + [(n, "gather:1:128") for n in range(2, 7)]
DG += [(n, v) for n in (3, 6, 11) for v in ("eo", "gather", "eof")]


@pytest.mark.parametrize("chunks", [8, 16])
@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("n,variant", DG)
def test_conforming_mesh(monkeypatch, n, variant, steps, chunks):
    """A single step starts by element lists of several groups (tcl: two CTAs an entry)."""
    monkeypatch.setenv("NMG_COPY_CHUNKS", str(chunks))
    _equal(_mesh("shells", n, 1), variant, 1e-3, steps)
    _equal(_mesh("box", n, 2), variant, 1e-3, steps)


@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("n,luni", [(9, 3), (6, 3)])
def test_conforming_mesh_by_size(n, luni, steps):
    """3584 elements: eight and three chunks by the size rule."""
    _equal(_mesh("shells", n, luni), "tc", 1e-3, steps)


@pytest.mark.parametrize("chunks", [2, 8])
@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("n,variant", [(n, v) for n, v in DG if n > 3])
def test_refined_mesh(monkeypatch, n, variant, steps, chunks):
    """Non-conforming faces: only the last stage runs in chunks."""
    monkeypatch.setenv("NMG_COPY_CHUNKS", str(chunks))
    _equal(_mesh("shells", n, 1, hrefine=(0, 3)), variant, 1e-3, steps)
