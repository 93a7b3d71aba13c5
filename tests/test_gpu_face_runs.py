"""The FP64 face runs of the transport tile (WENO without a division per weight) at the
edges of their ranges: extents around the tile and run lengths, fields that are zero,
tiny or uniform, and values beyond the scaled evaluation's range (taken again with a
scale per centre), against the oracle.  Tolerance: 1e-12 of the gross magnitude of the
terms summed into dsdt, as for the other FP64 updates."""
import numpy as np
import pytest
import torch

import oracle
from tests._util import scaled_err
from vidyut_b200 import _abi as abi
from vidyut_b200 import api
from vidyut_b200 import inputs as vin
from vidyut_b200 import mechanism as mm

pytestmark = pytest.mark.gpu

SIZES = [(1, (7,)), (1, (257,)), (2, (31, 9)), (2, (33, 8)), (3, (8, 8, 8)), (3, (9, 7, 17))]
FIELDS = ["rough", "tiny", "uniform", "zero", "huge"]


@pytest.mark.parametrize("dim,n", SIZES)
@pytest.mark.parametrize("field", FIELDS)
@pytest.mark.parametrize("hw", [(5, 1), (5, 2), (5, 3), (2, 3), (1, 3)])
def test_face_runs(dim, n, field, hw):
    mech = mm.synthetic(8, 40, vin.BASE_SEED + 21)
    case = vin.build_case(mech, dim, n, (1e-5, 2e-5, 1.5e-5)[:dim], vin.BASE_SEED + 301, density="loguniform",
                          dens_range=(1e10, 1e18), te_range_ev=(0.3, 10.0))
    ns = mech.ns
    sp = [s for s in range(ns + 1) if s not in mech.bg_species]
    if field == "tiny":  # eps of the smoothness indicators dominates
        case.state[sp] *= 1e-25
    elif field == "uniform":
        case.state[sp] = 1e12
    elif field == "zero":
        case.state[sp] = 0.0
    elif field == "huge":  # some cells beyond 4e32
        case.state[sp] *= 1e22
    prm = case.vd_params(hyp_order=hw[0], weno_scheme=hw[1], do_reactions=0, elecenergy_solve=1, do_transport=1,
                         const_ele_trans=1)
    api.mech_init(mech)
    dc = api.upload(case)
    phi_new, dsdt, _ = dc.new_outputs()
    api.explicit_update_all(dc, prm, phi_new, dsdt)
    torch.cuda.synchronize()
    port = oracle.Port(mech)
    want = port.update_all(case, prm)
    got = dsdt.cpu().numpy()
    assert np.isfinite(want["dsdt"]).all()
    assert scaled_err(got, want["dsdt"], port.update_scale(case, prm)) <= 1e-12
