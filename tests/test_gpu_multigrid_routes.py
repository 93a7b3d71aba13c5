"""Every route of the two multigrids: all levels in one CTA, levels by legs (2-D) and by
separate kernels (3-D rows of whole 16-byte groups and others), single-level hierarchies
and bottom grids of different sizes, at extents around the tiles' edges.  The potential
is checked against the solution by eigenvectors of the same discrete problem, the
species solve against its direct solve (oracle/diffusion.py).  Tolerances: the solvers
stop at a relative residual of 1e-11 / 1e-13, the solutions agree to 1e-9 / 1e-10 as in
the other tests of these solves; a single-level hierarchy does not converge in general,
so there only the residual reported is checked."""
import numpy as np
import pytest
import torch

import oracle
from oracle import diffusion as odf
from oracle import poisson as opois
from vidyut_b200 import _abi as abi
from vidyut_b200 import api, inputs
from vidyut_b200 import mechanism as mm

pytestmark = pytest.mark.gpu

V = 700.0


@pytest.fixture(scope="module")
def mech():
    m = mm.argon(10, 20261204)
    api.mech_init(m)
    return m


def eigen_solve(rhs, dx, vl):
    """The potential with vl and 0 at the x faces and zero gradient elsewhere."""
    nz, ny, nx = rhs.shape
    b = rhs.copy()
    b[:, :, 0] -= 2.0 * vl / dx[0] ** 2
    q, lam = [], []
    for d, n in enumerate((nx, ny, nz)):
        i = np.arange(n)
        k = i + 1 if d == 0 else i
        ang = np.pi * k[:, None] * (i[None, :] + 0.5) / n
        m = np.sin(ang) if d == 0 else np.cos(ang)
        q.append(m / np.linalg.norm(m, axis=1, keepdims=True))
        lam.append(-4.0 / dx[d] ** 2 * np.sin(np.pi * k / (2 * n)) ** 2 if n > 1 else np.zeros(1))
    c = np.einsum("kz,jy,ix,zyx->kji", q[2], q[1], q[0], b, optimize=True)
    c /= lam[2][:, None, None] + lam[1][None, :, None] + lam[0][None, None, :]
    return np.einsum("kz,jy,ix,kji->zyx", q[2], q[1], q[0], c, optimize=True)


@pytest.mark.parametrize("n", [(20, 16), (34, 32), (64, 48), (72, 40), (136, 96), (32, 32, 32), (36, 28, 28),
                               (34, 30, 28), (64, 48, 16)])
def test_potential(mech, n):
    dim = len(n)
    c = inputs.build_case(mech, dim, n, (1e-5,) * dim, 77 + sum(n), density="loguniform_smooth", dens_range=(1e14, 1e17),
                          te_range_ev=(0.5, 5.0))
    dc = api.upload(c)
    cyc, rr = api.poisson_solve(dc, c.vd_params(), api.poisson_params(dim, V, 0.0, max_vcycles=200, tol_rel=1e-11))
    g, v = c.gvec, c.n
    sl = (slice(g[2], g[2] + v[2]), slice(g[1], g[1] + v[1]), slice(g[0], g[0] + v[0]))
    rhs = -opois.ECHARGE / opois.EPS0 * sum(mech.charge[s] * c.state[s][sl] for s in range(mech.ns))
    want = eigen_solve(rhs, c.dx, V)
    got = dc.state[abi.POT(mech.ns)].cpu().numpy()[sl]
    assert 0 < cyc <= 200 and rr <= 1e-11
    assert np.max(np.abs(got - want)) <= 1e-9 * np.max(np.abs(want))


@pytest.mark.parametrize("n", [(301,), (21, 17), (41, 37), (15, 13, 11)])
def test_potential_single_level(mech, n):
    dim = len(n)
    c = inputs.build_case(mech, dim, n, (1e-5,) * dim, 177 + sum(n), density="loguniform_smooth",
                          dens_range=(1e14, 1e17), te_range_ev=(0.5, 5.0))
    r = []
    for cycles in (1, 40):
        dc = api.upload(c)
        r.append(api.poisson_solve(dc, c.vd_params(), api.poisson_params(dim, V, 0.0, max_vcycles=cycles, tol_rel=1e-300))[1])
    assert 0 <= r[1] < r[0]


@pytest.mark.parametrize("n", [(300,), (20, 16), (34, 32), (64, 48), (72, 40), (21, 17), (35, 34), (16, 12, 8),
                               (20, 16, 16), (22, 18, 14)])
@pytest.mark.parametrize("spec,walls", [(0, abi.BC_HNEU), (4, abi.BC_IHNEU)])
def test_species(mech, n, spec, walls):
    dim = len(n)
    dt = 1e-12 if walls == abi.BC_IHNEU else 1e-9
    bc = [[walls] * 3 for _ in range(4)]
    c = inputs.build_case(mech, dim, n, (1e-5,) * dim, 277 + sum(n), density="loguniform_smooth",
                          dens_range=(1e14, 1e18), te_range_ev=(0.5, 5.0))
    prm = c.vd_params(dt=dt, bc_lo=bc, bc_hi=bc, bound_specden=1)
    rng = np.random.default_rng(5)
    ns = mech.ns
    old = c.state.copy()
    old[:ns + 1] *= 1.0 + 0.01 * rng.uniform(-1, 1, old[:ns + 1].shape)
    g = c.gvec
    v = c.state[:, g[2]:g[2] + c.n[2], g[1]:g[1] + c.n[1], g[0]:g[0] + c.n[0]]
    dsdt = np.ascontiguousarray(1e-3 * v[:ns + 1] / dt * rng.uniform(-1, 1, v[:ns + 1].shape))
    dc = api.upload(c)
    phi_new = dc.new_outputs()[0]
    cyc, rr = api.implicit_species_solve(dc, spec, torch.from_numpy(old).cuda(), torch.from_numpy(dsdt).cuda(), phi_new,
                                         prm, tol_rel=1e-13, max_vcycles=200)
    assert 0 < cyc <= 200 and rr <= 1e-13
    sol = odf.solve(c, spec, old, dsdt[spec], prm, oracle.Port(mech))[0]
    got = phi_new[spec].cpu().numpy()
    if spec == ns:  # cells whose Te the floor raised hold the floor's energy
        keep = phi_new[ns + 1].cpu().numpy() > prm.min_electron_temp
        got, sol = np.where(keep, got, 0.0), np.where(keep, sol, 0.0)
    assert np.max(np.abs(got - sol)) <= 1e-10 * np.max(np.abs(sol))
