"""The two-kernel right-hand side of hexahedra against the gradient, node-flux
and surface passes (``ns_operator(..., return_gradients=True)`` takes those), on
meshes whose element counts leave a ragged last tile, with prescribed and dummy
boundary faces, anisotropic cells and every inviscid flux.  Both evaluate the
same float64 expressions in different orders: |difference| is bounded per field
by a few hundred roundings of the field's flux over the cell size."""

import numpy as np
import pytest
import torch

from cases import assert_fields_close, inviscid_flux_floor, make_disc, perturbed_state_np
from mirgecom_b200 import runtime
from mirgecom_b200.boundary import DummyBoundary, PrescribedFluidBoundary
from mirgecom_b200.eos import IdealSingleGas
from mirgecom_b200.fluid import ConservedVars
from mirgecom_b200.gas_model import GasModel, make_fluid_state
from mirgecom_b200.inviscid import (inviscid_facial_flux_central, inviscid_facial_flux_hll,
                                    inviscid_facial_flux_rusanov)
from mirgecom_b200.navierstokes import ns_operator
from mirgecom_b200.transport import SimpleTransport

pytestmark = pytest.mark.gpu

FLUX = {"rusanov": inviscid_facial_flux_rusanov, "hll": inviscid_facial_flux_hll,
        "central": inviscid_facial_flux_central}
TOL = 400 * 2.0 ** -53


@pytest.mark.parametrize("order,flux", [(1, "rusanov"), (2, "hll"), (3, "central"),
                                        (4, "rusanov"), (4, "hll")])
def test_matches_split_passes(cuda, order, flux):
    box = (1.0, 0.7, 1.3)
    d, od = make_disc("hypercube", 3, 3, order, (0.0,) * 3, box, False)
    q = perturbed_state_np(od.nodes, 3, 0, seed=order)
    qext = perturbed_state_np(od.nodes, 3, 0, seed=order + 20)
    gas = GasModel(eos=IdealSingleGas(), transport=SimpleTransport(
        viscosity=2e-2, thermal_conductivity=3e-2))

    def exterior(dcoll, dd_bdry, gas_model, state_minus, nodes=None, **kwargs):
        qb = state_minus.cv.q * 1.01
        return make_fluid_state(ConservedVars(qb, 3), gas_model)

    with pytest.warns(UserWarning):
        dummy = DummyBoundary()
    bnds = {"-0": PrescribedFluidBoundary(boundary_state_func=exterior), "+0": dummy,
            "-1": dummy, "+1": PrescribedFluidBoundary(boundary_state_func=exterior),
            "-2": dummy, "+2": dummy}
    st = make_fluid_state(ConservedVars(torch.from_numpy(q + 0.1 * qext).to(cuda), 3), gas)
    two = ns_operator(d, gas, st, bnds, inviscid_numerical_flux_func=FLUX[flux])
    split = ns_operator(d, gas, st, bnds, inviscid_numerical_flux_func=FLUX[flux],
                        return_gradients=True)[0]
    assert runtime.read_status(d) == 0
    floor = inviscid_flux_floor(st.cv.q.cpu().numpy(), 3, min(box) / 3 / order ** 2)
    assert_fields_close(two.q.cpu().numpy(), split.q.cpu().numpy(), TOL, floor=floor)
