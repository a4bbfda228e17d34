"""con2prim as the GRHD stages run it (c2p_fast, its own formula of the pressure function)
at the edges: data that are not numbers, no density, negative energy, momentum beyond the
energy, the points of the atmosphere and those an ulp beside them, guesses of every kind,
fast flow.  Against the oracle's pointwise con2prim: the same points are reset, to the same
state, and the others agree to what the root's condition leaves of FP64: p follows from E = rho h
W^2 - p by a difference with relative condition W^2 rho h / p, and W takes another W^2."""
import numpy as np
import pytest

import nmesh_gb300 as ng
from oracle import nmo

pytestmark = pytest.mark.gpu

N, NDIV = 7, 2
GAMMA, RHO_ATM, P_ATM = 2.0, 1e-10, 1e-18
EPS = 2.0 ** -53


@pytest.fixture(autouse=True)
def _gpu(cuda_ok):
    yield


def _spoil(kind, u, guess, ps, rng):
    npts = ps.size
    if kind == "not numbers":
        bad = np.nonzero(rng.random(npts) < 0.3)[0]
        u[rng.integers(0, 5, bad.size), bad] = rng.choice([np.nan, np.inf, -np.inf], bad.size)
    elif kind == "no density":
        u[0] *= rng.choice([-1.0, 0.0, 1e-12], npts)
    elif kind == "negative energy":
        u[4] *= -10.0 ** rng.uniform(-6, 0.5, npts)
    elif kind == "momentum beyond the energy":
        # above tau + D; a trace up to ten times it
        u[1:4] *= (u[4] + u[0]) * ps ** 2 / np.sqrt((u[1:4] ** 2).sum(0)) * 10.0 ** rng.uniform(-1e-3, 1, npts)
    elif kind in ("atmosphere at rest", "atmosphere moving"):
        ps6 = ps * ps * ps * ps * ps * ps
        u[0] = ps6 * RHO_ATM * (1 + rng.integers(-3, 4, npts) * 2.0 ** -52)
        tau_atm = RHO_ATM * (1 + P_ATM / RHO_ATM + P_ATM / RHO_ATM) - P_ATM
        u[4] = ps6 * tau_atm - u[0]
        u[1:4] = 0
        guess[:] = 0
        guess[0], guess[4] = RHO_ATM, P_ATM
        if kind == "atmosphere moving":
            u[1:4] = 1e-14 * rng.standard_normal((3, npts))
            u[4] = 10.0 ** rng.uniform(-14, -9, npts)
    elif kind == "guesses":
        guess[4] = rng.choice([np.nan, np.inf, -1.0, 0.0, 1e30, 1e-300], npts)


@pytest.mark.parametrize("mass", [0.0, 1.0])
@pytest.mark.parametrize("kind", ["plain", "fast", "not numbers", "no density", "negative energy",
                                  "momentum beyond the energy", "atmosphere at rest",
                                  "atmosphere moving", "guesses"])
def test_edges_like_the_pointwise_oracle(kind, mass):
    eos = dict(gamma=GAMMA, rho_atm=RHO_ATM, p_atm=P_ATM, tol=1e-15, maxits=100)
    m = ng.Mesh.build(ng.MESH_CUBEDSHELL6, n=N, ndiv=NDIV, shell_rin=2.0, shell_rout=20.0)
    ev = ng.GrhdEvolution(m, nf=13, mass=mass, **eos)
    x = m.coords()
    ps = (1.0 + 0.5 * mass / np.sqrt(x[:, 0] * x[:, 0] + x[:, 1] * x[:, 1] + x[:, 2] * x[:, 2])).reshape(-1)
    rng = np.random.default_rng(len(kind))
    rho = 10.0 ** rng.uniform(-8, 0, ps.size)
    p = rho * 10.0 ** rng.uniform(-4, 1, ps.size)
    W = 1 + 10.0 ** rng.uniform(-4, 2 if kind == "fast" else 0.5, ps.size)
    v = rng.standard_normal((3, ps.size))
    v *= np.sqrt(1 - 1 / W ** 2) / np.linalg.norm(v, axis=0) / ps ** 2
    prim = np.stack([rho, v[0], v[1], v[2], p])
    u = nmo.grhd_prim2con(prim, ps)
    guess = prim.copy()
    guess[4] *= rng.uniform(0.5, 1.5, ps.size)
    with np.errstate(invalid="ignore"):
        _spoil(kind, u, guess, ps, rng)

    def rows(a):
        return a.reshape(5, m.nelem, -1).transpose(1, 0, 2)

    empty = np.zeros((0, 5, 13 ** 3))
    ev.set_state(rows(u), empty, rows(guess), empty)
    ev.reset_stats()
    ev.rhs()
    got_u, _, got_p, _ = (a.transpose(1, 0, 2).reshape(5, -1) for a in ev.get_state())
    want_p, want_u, status = nmo.grhd_con2prim(u, guess, ps, **eos)
    reset = status < 0
    assert ev.stats()[1] == reset.sum()
    atm = (got_p[0] == RHO_ATM) & (got_p[4] == P_ATM) & (got_p[1:4] == 0).all(0)
    assert atm[reset].all()
    assert np.abs(got_u[:, reset] - want_u[:, reset]).max(initial=0) <= 4 * EPS * (ps ** 6).max() * RHO_ATM
    assert np.isfinite(got_p).all() and np.array_equal(got_u[:, ~reset], u[:, ~reset])
    ok = ~reset
    if kind.startswith("atmosphere"):
        assert kind != "atmosphere at rest" or 0 < reset.sum() < ps.size
        assert np.abs(got_p[:, ok] - want_p[:, ok]).max(initial=0) <= 4 * EPS * RHO_ATM
        return
    assert reset.all() or reset.sum() < 0.4 * ps.size
    h = rho + GAMMA / (GAMMA - 1) * p
    tol = 50 * EPS * (W ** 4 * h / p)[ok]
    for f in (0, 4):
        assert (np.abs(got_p[f] - want_p[f])[ok] <= tol * want_p[f][ok]).all(), f
