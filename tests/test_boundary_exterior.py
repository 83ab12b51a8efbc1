"""Boundary data handed to ``exterior_state`` (``runtime.boundary_exterior``):
the coordinates and unit normals are the callee's own, a call that changes them
in place changes no later call (host side, CPU tensors); and the data kept per
tag are complete for every stream once they are kept (GPU)."""

import numpy as np
import pytest
import torch

from cases import make_disc, perturbed_state_np
from mirgecom_b200 import runtime
from mirgecom_b200.boundary import PrescribedFluidBoundary
from mirgecom_b200.eos import IdealSingleGas
from mirgecom_b200.fluid import ConservedVars
from mirgecom_b200.gas_model import GasModel, make_fluid_state

TAGS = ("-0", "+0", "-1", "+1", "-2", "+2")


class _InPlace(PrescribedFluidBoundary):
    """Outflow along the normal that works in the arrays it is given."""

    def __init__(self):
        super().__init__(boundary_state_func=lambda **kwargs: None)
        self.seen = []

    def exterior_state(self, dcoll, dd_bdry, gas_model, state_minus, time, nodes=None,
                       normals=None):
        self.seen.append((nodes.clone(), normals.clone()))
        nodes.mul_(2.0).add_(1.0)
        normals.mul_(-3.0)
        q = state_minus.cv.q.clone()
        q[2:2 + state_minus.dim] += normals * nodes
        return make_fluid_state(ConservedVars(q, state_minus.dim), gas_model)


@pytest.mark.parametrize("kind,dim", [("simplex", 2), ("simplex", 3), ("hypercube", 3)])
@pytest.mark.parametrize("per_side", [False, True])
def test_callbacks_own_their_nodes_and_normals(kind, dim, per_side):
    d, od = make_disc(kind, dim, 3, 2, (0.0,) * dim, (1.0, 0.8, 1.2)[:dim], False)
    gas = GasModel(eos=IdealSingleGas())
    q = torch.from_numpy(perturbed_state_np(od.nodes, dim, 0, seed=4))
    st = make_fluid_state(ConservedVars(q, dim), gas)
    dd = runtime.DeviceDiscretization(d, torch.device("cpu"))
    bdry = _InPlace()
    tags = TAGS[:2 * dim] if per_side else ("all",)
    first = runtime.boundary_exterior(dd, st, gas, {t: bdry for t in tags}, 0.0)[:-1].clone()
    again = runtime.boundary_exterior(dd, st, gas, {t: bdry for t in tags}, 0.0)[:-1]
    assert torch.equal(first, again)
    for i, tag in enumerate(2 * tags):
        mask = d.boundary_face_mask(tag)
        nodes, normals = bdry.seen[i]
        np.testing.assert_array_equal(nodes.numpy(), d.boundary_nodes_numpy()[:, mask])
        np.testing.assert_array_equal(normals[:, :, 0].numpy(),
                                      d.boundary_normals_numpy()[mask].T)


@pytest.mark.gpu
def test_tag_data_are_complete_for_other_streams(cuda):
    """Kept while the first caller's stream is busy, read on another one."""
    d, _ = make_disc("simplex", 3, 4, 2, (0.0,) * 3, (1.0, 0.8, 1.2), False)
    dd = runtime.device_discretization(d, cuda)
    torch.cuda.synchronize()
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(200_000_000)                     # about 0.1 s
        for tag in TAGS:
            dd.boundary_tag(tag)
    c = d.connectivity
    with torch.cuda.stream(other):
        for tag in TAGS:
            got = [v.cpu().numpy() for v in dd.boundary_tag(tag)]
            mask = d.boundary_face_mask(tag)
            want = (np.nonzero(mask)[0], c.bface_elem[mask][:, None],
                    d.refel.face_nodes[c.bface_face[mask]], d.boundary_nodes_numpy()[:, mask],
                    d.boundary_normals_numpy()[mask].T[:, :, None])
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g, w)
    torch.cuda.synchronize()
