"""The per-call kernels at the edges of their tiles: face fluxes (tiles of 32 x 8, 8 x 32
and, with many tiles, 16 x 32 faces), the Joule term (tiles with a ring of density sums)
and the generated reaction source against the table-driven one, which it equals bit for
bit.  FP64 tolerance 1e-12 of the largest value, as the other per-call tests."""
import numpy as np
import pytest
import torch

import oracle
from tests._util import normwise_rel
from vidyut_b200 import _abi as abi
from vidyut_b200 import api
from vidyut_b200 import inputs as vin
from vidyut_b200 import mechanism as mm

pytestmark = pytest.mark.gpu

SIZES = [(1, (31,)), (1, (257,)), (2, (33, 9)), (2, (32, 8)), (2, (520, 305)), (3, (33, 17, 9)), (3, (40, 33, 20)),
         (3, (8, 8, 4))]


def _case(dim, n):
    return vin.build_case(mm.synthetic(8, 40, vin.BASE_SEED + 21), dim, n, (1e-5, 2e-5, 1.5e-5)[:dim],
                          vin.BASE_SEED + 401, density="loguniform", dens_range=(1e10, 1e18))


@pytest.mark.parametrize("dim,n", SIZES)
def test_face_flux_tiles(dim, n):
    case = _case(dim, n)
    m = case.mech
    api.mech_init(m)
    dc = api.upload(case)
    port = oracle.Port(m)
    for s in (m.e_id, 2, m.ns):  # electrons, a species without drift, the electron energy
        for d in range(dim):
            for h, w in ((5, 3), (2, 3), (1, 3)):
                fx = api.face_tensor(case, d)
                api.compute_explicit_flux(dc, d, s, fx, hyp_order=h, weno=w)
                assert normwise_rel(fx.cpu().numpy(), port.flux(case, d, s, hyp_order=h, weno=w)) <= 1e-12, (s, d, h)


@pytest.mark.parametrize("dim,n", [s for s in SIZES if s[1] != (520, 305)])
def test_joule_and_source_tiles(dim, n):
    case = _case(dim, n)
    m = case.mech
    api.mech_init(m)
    dc = api.upload(case)
    port = oracle.Port(m)
    rxn_np = port.reaction_source(case)
    prm = case.vd_params()
    de_want, pn_want = port.elecenergy(case, rxn_np, prm)
    phi_new, _, rxn = dc.new_outputs()
    de = torch.zeros((1, case.n[2], case.n[1], case.n[0]), dtype=torch.float64, device="cuda")
    api.compute_elecenergy_source(dc, torch.from_numpy(rxn_np).cuda(), de, phi_new, prm)
    assert normwise_rel(de.cpu().numpy(), de_want) <= 1e-12
    assert normwise_rel(phi_new.cpu().numpy()[abi.EJH(m.ns)], pn_want[abi.EJH(m.ns)]) <= 1e-12
    api.reaction_source(dc, rxn)
    L = abi.lib()
    try:
        L.vd_set_specialize(0)
        api.mech_init(m)
        table = torch.zeros_like(rxn)
        api.reaction_source(dc, table)
    finally:
        L.vd_set_specialize(1)
        api.mech_init(m)
    assert torch.equal(rxn, table)
