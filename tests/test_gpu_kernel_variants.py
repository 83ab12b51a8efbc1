"""Edges of the right-hand-side kernels' variants.

* tcgen05 gradients at order 2 (two row blocks of eight elements, rows moved
  in 8-byte pieces), against the mma.sync kernel and the float64 gradients,
  as test_gpu_grad_tc.py does for orders 1 and 3;
* the flux-volume kernel's inputs: rows off 16-byte boundaries are read from
  global memory instead of staged by bulk copies, with identical results; a
  partition whose last tile's rows end off 16 bytes;
* the mixture temperature from one polynomial pair per node against the
  species sums (which mechanisms with differing mid temperatures take), with
  iterations that cross the mid temperature.
"""

import copy

import numpy as np
import pytest
import torch

from cases import assert_fields_close, inviscid_flux_floor, make_disc, perturbed_state_np
from mirgecom_b200 import runtime
from mirgecom_b200.eos import IdealSingleGas, PyrometheusMixture
from mirgecom_b200.fluid import ConservedVars
from mirgecom_b200.gas_model import GasModel, make_fluid_state
from mirgecom_b200.initializers import reacting_mixture_state
from mirgecom_b200.navierstokes import ns_operator
from mirgecom_b200.thermochemistry import UIUC_7SP
from mirgecom_b200.transport import SimpleTransport
from test_gpu_grad_tc import _check, _mixture

pytestmark = pytest.mark.gpu

BOX = (0.02, 0.014, 0.026)


def _gas(mech=UIUC_7SP):
    return GasModel(eos=PyrometheusMixture(mech, temperature_niter=5),
                    transport=SimpleTransport(viscosity=2e-5, thermal_conductivity=3e-2,
                                              species_diffusivity=[1e-5] * 7))


@pytest.mark.parametrize("n", [3, 5])
def test_gradient_tc_order2(cuda, n):
    d, od = make_disc("simplex", 3, n, 2, (0.0,) * 3, BOX, True)
    gas, st64, st32 = _mixture(d, od, cuda, BOX, seed=n)
    _check(d, gas, st64, st32, {}, min(BOX) / n)


def _offset_copy(t):
    """The same values one element past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 2, dtype=t.dtype, device=t.device)
    out = buf[1:1 + t.numel()].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 != 0
    return out


@pytest.mark.parametrize("dim,order", [(2, 1), (2, 3), (3, 1), (3, 2), (3, 3)])
def test_flux_rows_off_16_bytes(cuda, dim, order):
    d, od = make_disc("simplex", dim, 3, order, (0.0,) * dim, BOX[:dim], True)
    cv0, t = reacting_mixture_state([torch.from_numpy(od.nodes[i]) for i in range(dim)], UIUC_7SP,
                                    seed=2, t_range=(900.0, 1500.0), box=BOX[:dim])
    gas = _gas()
    out = []
    for place in (lambda x: x, _offset_copy):
        cv = ConservedVars(place(cv0.q.to(cuda)), dim)
        st = make_fluid_state(cv, gas, temperature_seed=(t + 3.0).to(cuda))
        out.append(ns_operator(d, gas, st, {}, species_source_temperature=st.temperature).q)
    assert runtime.read_status(d) == 0
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("dim,order", [(2, 1), (2, 2), (2, 4), (3, 1), (3, 2), (3, 3)])
def test_flux_rows_off_16_bytes_float32(cuda, dim, order):
    """Every input row off 16 bytes, at 4, 8 or 12 bytes of it; the mma.sync
    gradient kernel on both sides, so that the gradients are the same."""
    d, od = make_disc("simplex", dim, 4, order, (0.0,) * dim, BOX[:dim], True)
    assert d.nelements * d.refel.nnodes % 4 == 0
    cv0, t = reacting_mixture_state([torch.from_numpy(od.nodes[i]) for i in range(dim)], UIUC_7SP,
                                    seed=2, t_range=(900.0, 1500.0), box=BOX[:dim])
    gas = _gas()
    q = cv0.q.to(cuda, torch.float32).contiguous()
    out = []
    runtime.set_gradient_kernel("mma_sync")
    try:
        for off in (0, 1, 2, 3):
            buf = torch.empty(q.numel() + 4, dtype=q.dtype, device=cuda)
            qo = buf[off:off + q.numel()].view(q.shape)
            qo.copy_(q)
            assert qo.data_ptr() % 16 == 4 * off
            st = make_fluid_state(ConservedVars(qo, dim), gas,
                                  temperature_seed=(t + 3.0).to(cuda, torch.float32))
            out.append(ns_operator(d, gas, st, {}, species_source_temperature=st.temperature).q)
    finally:
        runtime.set_gradient_kernel("auto")
    assert runtime.read_status(d) == 0
    for o in out[1:]:
        assert torch.equal(out[0], o)


@pytest.mark.parametrize("order", [1, 4])
def test_flux_rows_of_odd_2d_meshes_float32(cuda, order):
    """Rows whose pitch is off 16 bytes (an odd number of cells of odd-sized
    elements), against the float64 right-hand side at the mixed form's bar."""
    d, od = make_disc("simplex", 2, 5, order, (0.0,) * 2, (1.0, 0.7), True)
    assert d.nelements * d.refel.nnodes * 4 % 16 != 0
    q = perturbed_state_np(od.nodes, 2, 0, seed=order)
    gas = GasModel(eos=IdealSingleGas(),
                   transport=SimpleTransport(viscosity=2e-2, thermal_conductivity=3e-2))
    saved, out = runtime.RHS_PATH, []
    runtime.RHS_PATH = "gradient_volume_face"
    try:
        for dtype in (torch.float32, torch.float64):
            cv = ConservedVars(torch.from_numpy(q).to(cuda, dtype), 2)
            out.append(ns_operator(d, gas, make_fluid_state(cv, gas), {}).q)
    finally:
        runtime.RHS_PATH = saved
    assert runtime.read_status(d) == 0
    floor = inviscid_flux_floor(q, 2, 0.7 / 5 / order ** 2)
    assert_fields_close(out[0].double().cpu().numpy(), out[1].cpu().numpy(), 5e-5, floor=floor)


@pytest.mark.parametrize("order,elems,owned", [(2, 162, 61), (2, 162, 81), (1, 162, 61)])
def test_last_tile_off_16_bytes_float32(cuda, order, elems, owned):
    """The first *owned* of *elems* elements through the C entry point, float32:
    whole rows on 16 bytes, a last tile that ends off them (order 2, odd count),
    against the same elements of the whole mesh's flux-volume pass."""
    d, od = make_disc("simplex", 3, 3, order, (0.0,) * 3, BOX, True)
    assert d.nelements == elems
    cv0, t = reacting_mixture_state([torch.from_numpy(od.nodes[i]) for i in range(3)], UIUC_7SP,
                                    seed=2, t_range=(900.0, 1500.0), box=BOX)
    gas = _gas()
    st = make_fluid_state(ConservedVars(cv0.q.to(cuda, torch.float32).contiguous(), 3), gas,
                          temperature_seed=(t + 3.0).to(cuda, torch.float32))
    dd = runtime.device_discretization(d, cuda)
    out = []
    for n in (0, owned):
        dd.mesh.nowned = n
        try:
            rhs = torch.zeros_like(st.cv.q)
            runtime.ns_rhs(d, st, gas, {}, 0.0, 0, source_temperature=st.temperature, phases=1,
                           rhs=rhs)
            gs = runtime._gas_struct(gas, 7, cuda)
            out.append((rhs[:, :owned].clone(),
                        runtime.face_records(dd, gs, True, 12)[:owned].clone()))
        finally:
            dd.mesh.nowned = 0
    assert runtime.read_status(d) == 0
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-7)])
def test_temperature_polynomial_against_species_sums(cuda, dtype, tol):
    """1e-12: a hundred float64 roundings of energy terms up to ~50 c_v T;
    2e-7: the float32 temperature's last two bits."""
    g = torch.Generator().manual_seed(4)
    n = 4099
    x = [torch.rand(n, generator=g, dtype=torch.float64) * b for b in BOX]
    cv0, t = reacting_mixture_state(x, UIUC_7SP, seed=3, box=BOX)
    assert bool((t < 990).any()) and bool((t > 1010).any())
    # seeds on the other side of the mid temperature (1000 K) for many nodes
    seed = (t + 400.0 * (torch.rand(n, generator=g, dtype=torch.float64) - 0.5)).clamp(300, 2500)
    other = copy.deepcopy(UIUC_7SP)
    other.t_mid = UIUC_7SP.t_mid.copy()
    other.t_mid[-1] += 1e-9
    res = []
    for mech in (UIUC_7SP, other):
        gas = GasModel(eos=PyrometheusMixture(mech, temperature_niter=12))
        st = make_fluid_state(ConservedVars(cv0.q.to(cuda, dtype).contiguous(), 3), gas,
                              temperature_seed=seed.to(cuda, dtype))
        res.append(st.temperature.double().cpu().numpy())
    assert np.max(np.abs(res[0] - res[1]) / res[1]) < tol


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("cold", [False, True])
def test_learned_temperature_of_both_mechanism_forms(cuda, dim, cold):
    """The learned-guess kernel of a mechanism with one mid temperature (the
    polynomial pair) and of one without (species sums), warm warps and warps
    that run the network, a ragged last warp: 2e-7 of each other, two float32
    roundings of T (6e-8 each) and two accepted residuals (1e-8)."""
    from mirgecom_b200.learned_guess import TemperatureMLP
    g = torch.Generator().manual_seed(4)
    n = 4099
    x = [torch.rand(n, generator=g, dtype=torch.float64) * b for b in BOX[:dim]]
    cv0, t = reacting_mixture_state(x, UIUC_7SP, seed=3, box=BOX[:dim])
    other = copy.deepcopy(UIUC_7SP)
    other.t_mid = UIUC_7SP.t_mid.copy()
    other.t_mid[-1] += 1e-9
    net = TemperatureMLP(cuda, seed=0)
    e, y, tt = TemperatureMLP.training_pairs(UIUC_7SP, 1 << 13, cuda, seed=0)
    net.fit(e, y, tt, steps=100, batch=1 << 13, lr=3e-3, seed=0)
    res = []
    for mech in (UIUC_7SP, other):
        gas = GasModel(eos=PyrometheusMixture(mech, temperature_niter=12, learned_guess=net))
        st = make_fluid_state(ConservedVars(cv0.q.to(cuda, torch.float32).contiguous(), dim), gas,
                              temperature_seed=300.0 if cold else (t + 2.0).to(cuda, torch.float32))
        res.append(st.temperature.double().cpu().numpy())
    assert int(runtime.state_status_word(cuda).item()) == 0
    assert np.max(np.abs(res[0] - res[1]) / res[1]) < 2e-7
    # and of the temperatures the state was made from, to the float32 state's
    # roundings of the energy (formation enthalpies of ~1e7 J/kg over c_v T)
    assert np.max(np.abs(res[0] - t.numpy()) / t.numpy()) < 1e-4
