"""The work this library is used for, as cases that can be timed and checked.

Each case is one call (or one step) that a flow solver built on the library
makes, through the public entry points: the right-hand side of the Navier-Stokes
equations for the ideal gas and for the 7-species reacting mixture (float64 and
the mixed form), Euler and reacting Runge-Kutta steps, the mixture temperature
solve and one training step of the learned temperature guess.  Sizes are those
of the library's own configurations (the 2-D vortex, the Taylor-Green vortex on
tetrahedra and hexahedra, the reacting boxes at orders 2 and 3) and of its wall
tests; ``draw`` spreads over the ranges around them.

``prepare`` builds what a program holds before the call.  The mesh, its
discretization and the trained network are kept per process, as such a program
keeps them; the states are made from the seed.
"""

import functools
import math

import numpy as np
import torch

from mirgecom_b200.boundary import (AdiabaticNoslipWallBoundary, FarfieldBoundary,
                                    IsothermalWallBoundary, PrescribedFluidBoundary,
                                    PressureOutflowBoundary)
from mirgecom_b200.discretization import create_discretization_collection
from mirgecom_b200.eos import IdealSingleGas, PyrometheusMixture
from mirgecom_b200.euler import euler_operator
from mirgecom_b200.fluid import ConservedVars
from mirgecom_b200.gas_model import GasModel, make_fluid_state
from mirgecom_b200.initializers import (Vortex2D, reacting_mixture_state, taylor_green_state,
                                        taylor_green_transport_params)
from mirgecom_b200.integrators import rk4_step, rk4_step_mixed
from mirgecom_b200.inviscid import inviscid_facial_flux_hll, inviscid_facial_flux_rusanov
from mirgecom_b200.learned_guess import H, KIN, NPARAM, TemperatureMLP
from mirgecom_b200.mesh import generate_box_mesh
from mirgecom_b200.navierstokes import ns_operator
from mirgecom_b200.thermochemistry import GAS_CONSTANT, ONE_ATM, UIUC_7SP
from mirgecom_b200.transport import PowerLawTransport, SimpleTransport

FLUXES = {"rusanov": inviscid_facial_flux_rusanov, "hll": inviscid_facial_flux_hll}
WALL_CELL = 0.0065                     # cell size of the wall-bounded boxes, m
WALL_T, OUT_P = 1000.0, 101325.0       # isothermal walls, outflow pressure
FREE = dict(pressure=101325.0, velocity=[3.0, -1.0, 2.0], temperature=1200.0,
            fractions=[0.05, 0.22, 0.0, 0.0, 0.0, 0.0, 0.73])
SIMPLE = dict(mu=1e-5, kappa=1e-5, diff=1e-5)
POWER = dict(alpha=0.6, beta=4.093e-7, sigma=2.5, n=0.666)
DT_VORTEX, DT_REACTING = 0.005, 1e-9
LR, BETA1, BETA2, EPS = 1e-3, 0.9, 0.999, 1e-8


def _mesh_case(call, order, counts, gas="mixture", dtype="f64", elem="simplex", bc="periodic",
               flux="rusanov", transport="simple", guess="plain", seeds="warm"):
    n = list(counts) + [0] * (3 - len(counts))
    return dict(call=call, elem=elem, order=order, nx=n[0], ny=n[1], nz=n[2], gas=gas,
                dtype=dtype, bc=bc, flux=flux, transport=transport, guess=guess, seeds=seeds)


def listed():
    return [
        # one RK4 step of the 2-D isentropic vortex with the exact solution
        # prescribed on the boundary: the smallest mesh a driver steps
        # through, four small right-hand sides with their boundary callbacks
        dict(name="vortex2d_step", **_mesh_case("euler_step", 3, (16, 16), gas="ideal",
                                                bc="exact")),
        # Taylor-Green vortex on tetrahedra, float64: the single-gas viscous
        # right-hand side of a direct simulation at an ordinary size
        dict(name="tgv_p3_tet24", **_mesh_case("ns", 3, (24,) * 3, gas="ideal")),
        # the same flow on high-order hexahedra (sum-factorised kernels)
        dict(name="tgv_p4_hex48", **_mesh_case("ns", 4, (48,) * 3, gas="ideal",
                                               elem="hypercube")),
        # a small hexahedral mesh: a convergence study's coarse level
        dict(name="tgv_p2_hex10", **_mesh_case("ns", 2, (10, 9, 11), gas="ideal",
                                               elem="hypercube")),
        # reacting mixture, mixed form: per-device size of a strongly scaled
        # run (small), a mid-size order-2 mesh, and a large order-3 mesh with
        # the learned temperature guess
        dict(name="reacting_p3_tet6", **_mesh_case("ns", 3, (6, 7, 5), dtype="f32")),
        dict(name="reacting_p2_tet40", **_mesh_case("ns", 2, (40,) * 3, dtype="f32")),
        dict(name="reacting_p3_tet64", **_mesh_case("ns", 3, (64,) * 3, dtype="f32",
                                                    guess="learned")),
        # the plain float64 form of the reacting right-hand side
        dict(name="reacting_p3_tet32_f64", **_mesh_case("ns", 3, (32,) * 3)),
        # a wall-bounded reacting channel with gradients returned, HLL and
        # power-law transport; odd cell counts
        dict(name="channel_p2_tet13", **_mesh_case("ns_gradients", 2, (13, 9, 11), bc="walls",
                                                   flux="hll", transport="power")),
        # one mixed-precision RK4 step of the reacting mixture: what a
        # time-marching driver repeats
        dict(name="reacting_step_p3_tet20", **_mesh_case("reacting_step", 3, (20,) * 3,
                                                         dtype="f32", guess="learned")),
        # temperature of a state without a previous temperature (start-up,
        # restart): learned guess from the default cold seed
        dict(name="cold_temperature_p3_tet30", **_mesh_case(
            "temperature", 3, (30,) * 3, dtype="f32", guess="learned", seeds="cold")),
        # one training step (loss, gradients, Adam) of the learned guess
        dict(name="train_guess_64k", call="train", rows=65536),
    ]


# {{{ drawn cases

def _counts(rng, nodes, dim, per_cell):
    """Ragged cell counts with about *nodes* nodes in all."""
    n = (nodes / per_cell) ** (1.0 / dim)
    return tuple(max(4, round(n * math.exp(rng.uniform(-0.25, 0.25)))) for _ in range(dim))


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["vortex", "tgv", "hex", "reacting", "reacting", "reacting64", "channel",
                       "step", "temperature", "train"])
    p = rng.choice([1, 2, 3, 3])
    tet = 6 * (p + 1) * (p + 2) * (p + 3) // 6         # nodes per cell
    if kind == "vortex":
        p = rng.randint(1, 4)
        return _mesh_case("euler_step", p, _counts(rng, _log_uniform(rng, 2e3, 2e5), 2,
                                                   (p + 1) * (p + 2)), gas="ideal", bc="exact")
    if kind == "tgv":
        return _mesh_case("ns", p, _counts(rng, _log_uniform(rng, 2e4, 6e6), 3, tet),
                          gas="ideal", flux=rng.choice(["rusanov", "rusanov", "hll"]))
    if kind == "hex":
        p = rng.randint(1, 4)
        return _mesh_case("ns", p, _counts(rng, _log_uniform(rng, 2e4, 8e6), 3, (p + 1) ** 3),
                          gas="ideal", elem="hypercube")
    if kind == "reacting":
        return _mesh_case("ns", p, _counts(rng, _log_uniform(rng, 2e4, 1.5e7), 3, tet),
                          dtype="f32", guess=rng.choice(["plain", "learned"]),
                          transport=rng.choice(["simple", "simple", "power"]))
    if kind == "reacting64":
        return _mesh_case("ns", p, _counts(rng, _log_uniform(rng, 2e4, 4e6), 3, tet),
                          flux=rng.choice(["rusanov", "rusanov", "hll"]))
    if kind == "channel":
        return _mesh_case(rng.choice(["ns", "ns_gradients"]), p,
                          _counts(rng, _log_uniform(rng, 2e4, 5e5), 3, tet), bc="walls",
                          flux=rng.choice(["rusanov", "hll"]),
                          transport=rng.choice(["simple", "power"]))
    if kind == "step":
        return _mesh_case("reacting_step", p, _counts(rng, _log_uniform(rng, 2e4, 2e6), 3, tet),
                          dtype="f32", guess=rng.choice(["plain", "learned"]))
    if kind == "temperature":
        return _mesh_case("temperature", p, _counts(rng, _log_uniform(rng, 2e4, 5e6), 3, tet),
                          dtype="f32", guess="learned", seeds=rng.choice(["cold", "warm"]))
    return dict(call="train", rows=int(_log_uniform(rng, 2000, 250000)))

# }}}


# {{{ prepare and run

def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _box(case):
    """(lower corner, upper corner, cell counts, periodic) of the case's box."""
    n = tuple(int(case[k]) for k in ("nx", "ny", "nz") if case[k])
    if case["bc"] == "exact":
        return (0.0, -5.0), (10.0, 5.0), n, (False,) * 2
    if case["bc"] == "walls":
        return (0.0,) * 3, tuple(WALL_CELL * k for k in n), n, (False,) * 3
    if case["gas"] == "ideal":
        return (-math.pi,) * 3, (math.pi,) * 3, n, (True,) * 3
    return (0.0,) * 3, (2 * math.pi,) * 3, n, (True,) * 3


@functools.lru_cache(maxsize=3)
def _disc(elem, order, lo, hi, n, periodic):
    mesh = generate_box_mesh(lo, hi, n, kind=elem, periodic=periodic)
    return create_discretization_collection(mesh, order)


def _disc_of(case):
    return _disc(case["elem"], case["order"], *_box(case))


@functools.lru_cache(maxsize=1)
def _guess():
    dev = _device()
    net = TemperatureMLP(dev, seed=0)
    e, y, t = TemperatureMLP.training_pairs(UIUC_7SP, 1 << 18, dev, seed=0)
    net.fit(e, y, t, steps=1000, batch=65536, lr=3e-3, seed=0)
    return net


def _gas(case):
    if case["gas"] == "ideal":
        tr = None if case["call"] == "euler_step" else SimpleTransport(
            **taylor_green_transport_params())
        return GasModel(eos=IdealSingleGas(), transport=tr)
    tr = (PowerLawTransport(lewis=np.ones(7), **POWER) if case["transport"] == "power" else
          SimpleTransport(viscosity=SIMPLE["mu"], thermal_conductivity=SIMPLE["kappa"],
                          species_diffusivity=[SIMPLE["diff"]] * 7))
    learned = _guess() if case["guess"] == "learned" else None
    return GasModel(eos=PyrometheusMixture(UIUC_7SP, temperature_niter=5,
                                           learned_guess=learned), transport=tr)


def _vortex(seed):
    g = np.random.default_rng(seed)
    return Vortex2D(beta=g.uniform(4.0, 5.0), center=tuple(np.array([5.0, 0.0]) +
                                                           g.uniform(-0.5, 0.5, 2)),
                    velocity=tuple(np.array([1.0, 0.0]) + g.uniform(-0.2, 0.2, 2)))


def _inputs(case, seed, x, box):
    """(q, temperature seed): the float64 or float32 state on the nodes *x*."""
    dtype = torch.float32 if case["dtype"] == "f32" else torch.float64
    if case["bc"] == "exact":
        return _vortex(seed)(x).q, None
    if case["gas"] == "ideal":
        # the vortex array somewhere in its periodic box, at some strength
        g = np.random.default_rng(seed)
        cv = taylor_green_state([xi + float(s) for xi, s in zip(x, g.uniform(0, 6.28, 3))],
                                v0=float(g.uniform(0.8, 1.2)))
        return cv.q.to(dtype), None
    t_range = (900.0, 1500.0) if case["bc"] == "walls" else (300.0, 2500.0)
    cv, t = reacting_mixture_state(x, UIUC_7SP, seed=seed, t_range=t_range, box=box)
    # a warm seed is the temperature of the step before, a few kelvin off
    tseed = 300.0 if case["seeds"] == "cold" else t + 2.0
    if torch.is_tensor(tseed) and case["call"] != "reacting_step":
        tseed = tseed.to(dtype)
    return (cv.q if case["call"] == "reacting_step" else cv.q.to(dtype)).contiguous(), tseed


def _train_inputs(case, seed):
    dev = _device()
    e, y, t = TemperatureMLP.training_pairs(UIUC_7SP, int(case["rows"]), dev, seed=seed)
    net = TemperatureMLP(dev, seed=seed)
    net.set_normalisation(e, y)
    x = net.features(e, y)
    target = ((t.to(torch.float32) - net.out_shift) / net.out_scale).contiguous()
    # Adam moments as they are some way into the training
    g = torch.Generator(device=dev).manual_seed(seed)
    net.m.copy_(1e-3 * torch.randn(NPARAM, generator=g, device=dev))
    net.v.copy_(1e-4 + 1e-4 * torch.rand(NPARAM, generator=g, device=dev))
    net.step_count = 500
    return net, x, target


def prepare(case, seed):
    if case["call"] == "train":
        net, x, target = _train_inputs(case, seed)
        return dict(call="train", net=net, x=x, target=target)
    dcoll = _disc_of(case)
    lo, hi = _box(case)[:2]
    gas = _gas(case)
    x = dcoll.nodes(_device())
    q, tseed = _inputs(case, seed, x, [b - a for a, b in zip(lo, hi)])
    boundaries = {}
    if case["bc"] == "exact":
        init = _vortex(seed)

        def solution(dcoll, dd_bdry, gas_model, state_minus, time=0.0, nodes=None, **kwargs):
            xb = [nodes[i] for i in range(nodes.shape[0])]
            return make_fluid_state(init(xb, eos=gas_model.eos, time=time), gas_model)

        boundaries = {"all": PrescribedFluidBoundary(boundary_state_func=solution)}
    elif case["bc"] == "walls":
        far = FarfieldBoundary(FREE["pressure"], FREE["velocity"], FREE["temperature"],
                               FREE["fractions"])
        wall, noslip = IsothermalWallBoundary(WALL_T), AdiabaticNoslipWallBoundary()
        boundaries = {"-1": far, "+1": PressureOutflowBoundary(OUT_P), "-2": wall, "+2": wall,
                      "-3": noslip, "+3": noslip}
        boundaries = {t[0] + str(int(t[1]) - 1): b for t, b in boundaries.items()}
    return dict(call=case["call"], dcoll=dcoll, gas=gas, q=q, tseed=tseed,
                boundaries=boundaries, flux=FLUXES[case["flux"]])


def _ns(s, cv, gradients=False):
    st = make_fluid_state(cv, s["gas"], temperature_seed=s["tseed"])
    out = ns_operator(s["dcoll"], s["gas"], st, s["boundaries"],
                      inviscid_numerical_flux_func=s["flux"], return_gradients=gradients,
                      species_source_temperature=st.temperature if st.is_mixture else None)
    return st, out


def run(s):
    call = s["call"]
    if call == "train":
        loss, grad = s["net"].loss_and_grad(s["x"], s["target"])
        s["net"].adam_step(LR, BETA1, BETA2, EPS)
        return dict(loss=loss, grad=grad, params=s["net"].params)
    cv = ConservedVars(s["q"], s["dcoll"].dim)
    if call == "ns":
        st, rhs = _ns(s, cv)
        return dict(rhs=rhs.q, temperature=st.temperature) if st.is_mixture else dict(rhs=rhs.q)
    if call == "ns_gradients":
        st, (rhs, grad_cv, grad_t) = _ns(s, cv, gradients=True)
        return dict(rhs=rhs.q, grad_cv=grad_cv.q, grad_t=grad_t, temperature=st.temperature)
    if call == "temperature":
        return dict(temperature=make_fluid_state(cv, s["gas"],
                                                 temperature_seed=s["tseed"]).temperature)
    if call == "euler_step":
        def rhs(t, state):
            return euler_operator(s["dcoll"], make_fluid_state(state, s["gas"]), s["gas"],
                                  s["boundaries"], time=t,
                                  inviscid_numerical_flux_func=s["flux"])
        return dict(state=rk4_step(cv, 0.0, DT_VORTEX, rhs).q)
    new, new32 = rk4_step_mixed(cv, 0.0, DT_REACTING, lambda t, c: _ns(s, c)[1])
    return dict(state=new.q, state32=new32.q)


def work(case):
    """Inputs read once, outputs written once, and the contractions of the
    reference operators (dense on simplices, sum-factorised on hexahedra) with
    a count of the pointwise arithmetic: a flux evaluation per node, and for
    the mixture the NASA-7 and Arrhenius evaluations."""
    if case["call"] == "train":
        n = int(case["rows"])
        return dict(bytes=n * 9 * 4 + NPARAM * 6 * 4,
                    flops=3.0 * 2 * n * (H * 8 + H * H + H) + 10.0 * NPARAM)
    lo, _, n, _ = _box(case)
    d, p = len(lo), int(case["order"])
    cells = float(np.prod(n))
    hexes = case["elem"] == "hypercube"
    ne = cells if hexes else cells * math.factorial(d)
    npn = (p + 1) ** d if hexes else math.comb(p + d, d)
    nf = 2 * d if hexes else d + 1
    nfp = (p + 1) ** (d - 1) if hexes else math.comb(p + d - 1, d - 1)
    mix = case["gas"] == "mixture"
    nc, s = d + 2 + (7 if mix else 0), 4 if case["dtype"] == "f32" else 8
    nodes = ne * npn
    newton = nodes * 3 * 7 * 25.0 if mix else 0.0
    if case["call"] == "temperature":
        return dict(bytes=nodes * (nc + 1 + (case["seeds"] == "warm")) * s, flops=newton)
    line = 2.0 * (p + 3) if hexes else 2.0 * npn
    face = 0.0 if hexes else 2.0 * npn * nf * nfp
    div = ne * nc * (d * npn * line + face)
    grad = ne * (nc + 1) * (d * npn * line + face)
    point = nodes * (nc * d * 8.0 + (7 * 60.0 + 3 * 60.0 if mix else 20.0))
    geo = ne * (d * d * s + nf * 4)
    if case["call"] == "euler_step":
        return dict(bytes=nodes * 2 * nc * s + geo, flops=4 * (div + point))
    rhs = div + grad + point + newton
    if case["call"] == "reacting_step":
        return dict(bytes=nodes * (nc * (8 + 8 + 4) + 8) + geo, flops=4 * rhs)
    out = nc + (1 if mix else 0) + ((nc + 1) * d if case["call"] == "ns_gradients" else 0)
    return dict(bytes=nodes * (nc + (1 if mix else 0) + out) * s + geo, flops=rhs)

# }}}


# {{{ the same in 64 bits with plain torch

def _mech(name, like):
    return torch.as_tensor(np.asarray(getattr(UIUC_7SP, name)), dtype=torch.float64,
                           device=like.device)


def _col(v, like):
    return v.reshape((-1,) + (1,) * like.ndim)


def _nasa(t):
    """c_p/R, h/RT and s/R of every species at the temperatures *t*."""
    hi = t[None] > _col(_mech("t_mid", t), t)
    a_lo, a_hi = _mech("nasa_low", t), _mech("nasa_high", t)
    a = [torch.where(hi, _col(a_hi[:, j], t), _col(a_lo[:, j], t)) for j in range(7)]
    cp = a[0] + t * (a[1] + t * (a[2] + t * (a[3] + t * a[4])))
    h = a[0] + t * (a[1] / 2 + t * (a[2] / 3 + t * (a[3] / 4 + t * a[4] / 5))) + a[5] / t
    s = (a[0] * t.log() + t * (a[1] + t * (a[2] / 2 + t * (a[3] / 3 + t * a[4] / 4))) + a[6])
    return cp, h, s


class _Exact:
    """The discrete operators on the plan's mesh and reference matrices."""

    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        self.dev = _device() if torch.cuda.is_available() else torch.device("cpu")
        dc = self.dc = _disc_of(case)
        r, g, c = dc.refel, dc.geometry, dc.connectivity
        f64 = functools.partial(torch.as_tensor, dtype=torch.float64, device=self.dev)
        self.dim, self.mix = dc.dim, case["gas"] == "mixture"
        self.weak, self.lift, self.rx = f64(r.weak), f64(r.lift), f64(g.rx)
        self.nrm, self.fscale = f64(g.normals), f64(g.fscale)
        self.fn = torch.as_tensor(np.asarray(r.face_nodes), device=self.dev).long()
        self.nbr = torch.as_tensor(c.nbr_node_index, device=self.dev).long()
        self.be = torch.as_tensor(c.bface_elem, device=self.dev).long()
        self.bf = torch.as_tensor(c.bface_face, device=self.dev).long()
        self.side = torch.as_tensor(c.bface_side, device=self.dev).long()
        x = [f64(xi) for xi in g.nodes]
        lo, hi = _box(case)[:2]
        q, self.tseed = _inputs(case, seed, x, [b - a for a, b in zip(lo, hi)])
        self.q = q.double()
        self.bx = [xi[self.be[:, None], self.fn[self.bf]] for xi in x] if len(c.bface_elem) else []

    # gas
    def temperature(self, q, guess=None):
        rho, d = q[0], self.dim
        e = (q[1] - 0.5 * (q[2:2 + d] ** 2).sum(0) / rho) / rho
        if not self.mix:
            return 0.4 / 287.1 * e
        yw = q[2 + d:] / rho / _col(_mech("molecular_weights", rho), rho)
        t = torch.full_like(rho, 1200.0) if guess is None else guess.double()
        for _ in range(60):
            cp, h, _ = _nasa(t)
            dt = (e - GAS_CONSTANT * t * (yw * (h - 1)).sum(0)) / (
                GAS_CONSTANT * (yw * (cp - 1)).sum(0))
            t = (t + dt).clamp(150.0, 6000.0)
            if float((dt / t).abs().max()) < 1e-14:
                break
        return t

    def state(self, q, t):
        d, s = self.dim, {}
        s["q"], s["t"], s["rho"], s["v"] = q, t, q[0], q[2:2 + d] / q[0]
        s["y"] = q[2 + d:] / q[0]
        if self.mix:
            w = _col(_mech("molecular_weights", t), t)
            rmix = GAS_CONSTANT * (s["y"] / w).sum(0)
            cp_k, h_k, _ = _nasa(t)
            cp = GAS_CONSTANT * (s["y"] * cp_k / w).sum(0)
            s["h"] = GAS_CONSTANT * t * h_k / w
            s["p"], s["gamma"], s["cv"] = q[0] * rmix * t, cp / (cp - rmix), cp - rmix
        else:
            s["p"] = 0.4 * (q[1] - 0.5 * (q[2:2 + d] ** 2).sum(0) / q[0])
            s["gamma"], s["cv"] = torch.full_like(t, 1.4), 287.1 / 0.4
        s["c"] = (s["gamma"] * s["p"] / q[0]).sqrt()
        return s

    def energy(self, q, t):
        """Total energy density of the density, velocity and species of *q* at *t*."""
        d = self.dim
        yw = q[2 + d:] / q[0] / _col(_mech("molecular_weights", t), t)
        return (q[0] * GAS_CONSTANT * t * (yw * (_nasa(t)[1] - 1)).sum(0)
                + 0.5 * (q[2:2 + d] ** 2).sum(0) / q[0])

    def inviscid(self, s):
        d, q, v = self.dim, s["q"], s["v"]
        f = q[:, None] * v[None]
        f[1] = f[1] + s["p"] * v
        for i in range(d):
            f[2 + i, i] = f[2 + i, i] + s["p"]
        return f

    def viscous(self, s, gq, gt):
        d, rho, v, y = self.dim, s["rho"], s["v"], s["y"]
        if self.case["transport"] == "power" and self.mix:
            mu = POWER["beta"] * s["t"] ** POWER["n"]
            mub, kappa = POWER["alpha"] * mu, POWER["sigma"] * mu * s["cv"]
            diff = POWER["sigma"] * mu / (rho * s["gamma"])
        elif self.mix:
            mu, mub, kappa, diff = SIMPLE["mu"], 0.0, SIMPLE["kappa"], SIMPLE["diff"]
        else:
            par = taylor_green_transport_params()
            mu, mub, kappa, diff = par["viscosity"], 0.0, par["thermal_conductivity"], 0.0
        gv = (gq[2:2 + d] - v[:, None] * gq[0]) / rho
        div = sum(gv[i, i] for i in range(d))
        tau = mu * (gv + gv.transpose(0, 1))
        for i in range(d):
            tau[i, i] = tau[i, i] + (mub - 2.0 * mu / 3.0) * div
        f = torch.zeros_like(gq)
        f[2:2 + d] = tau
        f[1] = (tau * v[None]).sum(1) + kappa * gt
        if self.mix:
            gy = (gq[2 + d:] - y[:, None] * gq[0]) / rho
            flux = rho * (diff * gy - y[:, None] * (diff * gy).sum(0))
            f[2 + d:] = flux
            f[1] = f[1] + (s["h"][:, None] * flux).sum(0)
        return f

    def sources(self, q, t):
        w = _col(_mech("molecular_weights", t), t)
        conc = (q[2 + self.dim:] / w).clamp_min(0.0)
        _, h, s = _nasa(t)
        out = torch.zeros_like(conc)
        m = UIUC_7SP
        for i in range(m.nreactions):
            kf = torch.exp(m.log_a[i] + m.beta[i] * t.log() - m.t_act[i] / t)
            net = m.nu_prod[i] - m.nu_reac[i]
            rate = kf.clone()
            for k in np.nonzero(m.orders_fwd[i])[0]:
                rate = rate * conc[k] ** float(m.orders_fwd[i, k])
            if m.reversible[i]:
                dg = sum(float(net[k]) * (h[k] - s[k]) for k in np.nonzero(net)[0])
                back = kf * torch.exp(dg - float(net.sum()) * (
                    ONE_ATM / (GAS_CONSTANT * t)).log())
                for k in np.nonzero(m.nu_prod[i])[0]:
                    back = back * conc[k] ** float(m.nu_prod[i, k])
                rate = rate - back
            out = out + _col(torch.as_tensor(net, device=t.device), t) * rate
        return out * w

    # traces
    def inside(self, u):
        return u[..., self.fn]                              # [..., E, Nf, Nfp]

    def outside(self, u, bvals):
        """Neighbour values; *bvals* [..., nbf, Nfp] on the boundary faces."""
        up = u.flatten(-2)[..., self.nbr.clamp_min(0)]
        if bvals is not None and len(self.be):
            up[..., self.be, self.bf, :] = bvals
        return up

    def at_boundary(self, u):
        return u[..., self.be[:, None], self.fn[self.bf]]

    def boundary_states(self, q, t, time):
        """(state_plus, T; state_bc, T; temperature_bc) at the boundary nodes."""
        if not len(self.be):
            return None
        qm, tm = self.at_boundary(q), self.at_boundary(t)
        if self.case["bc"] == "exact":
            ext = _vortex(self.seed)(self.bx, time=time).q
            te = self.temperature(ext)
            return ext, te, ext, te, te
        qp, qb, tb = qm.clone(), qm.clone(), tm.clone()
        d = self.dim
        free = torch.zeros_like(qm)
        yf = torch.as_tensor(FREE["fractions"], dtype=torch.float64, device=self.dev)
        tf = torch.full_like(tm, FREE["temperature"])
        rho = FREE["pressure"] / (GAS_CONSTANT * (yf / _mech("molecular_weights", tm)).sum()
                                  * FREE["temperature"])
        free[0] = rho
        for i in range(d):
            free[2 + i] = rho * FREE["velocity"][i]
        free[2 + d:] = rho * yf[:, None, None]
        free[1] = self.energy(free, tf)
        sm = self.state(qm, tm)
        nrm = self.nrm[self.be, self.bf].T[:, :, None]
        sonic = (sm["v"] * nrm).sum(0).abs() > sm["c"]
        per_t = sm["p"] / tm                                # rho R_mix
        for side in range(6):
            on = (self.side == side)[:, None].expand_as(tm)
            if side == 0:
                for out in (qp, qb):
                    out.copy_(torch.where(on, free, out))
                tb = torch.where(on, tf, tb)
            elif side == 1:
                pp = torch.where(sm["p"] > 2 * OUT_P, sm["p"], 2 * OUT_P - sm["p"])
                for out, pr in ((qp, pp), (qb, torch.full_like(pp, OUT_P))):
                    en = self.energy(qm, torch.where(sonic, tm, pr / per_t))
                    out[1] = torch.where(on, en, out[1])
            else:
                tw = torch.full_like(tm, WALL_T) if side in (2, 3) else tm
                q0 = qm.clone()
                q0[2:2 + d] = 0
                q0[1] = self.energy(q0, tw)
                qb = torch.where(on, q0, qb)
                qp[2:2 + d] = torch.where(on, -qm[2:2 + d], qp[2:2 + d])
                tb = torch.where(on, tw, tb)
        return qp, self.temperature(qp, tm), qb, self.temperature(qb, tb), tb

    # operators
    def lifted(self, s):
        return torch.einsum("im,...em->...ei", self.lift,
                            (s * self.fscale[..., None]).flatten(-2))

    def gradient(self, u, ub):
        um = self.inside(u)
        up = self.outside(u, None)
        ustar = 0.5 * (um + up)
        if ub is not None:
            ustar[..., self.be, self.bf, :] = ub
        du = torch.einsum("rik,ek->rei", self.weak, u)
        vol = torch.einsum("erj,rei->jei", self.rx, du)
        return torch.stack([self.lifted(ustar * self.nrm[:, :, j, None])
                            for j in range(self.dim)]) - vol

    def gradients(self, q, t, bs):
        gq = torch.stack([self.gradient(q[c], None if bs is None else bs[2][c])
                          for c in range(q.shape[0])])
        return gq, self.gradient(t, None if bs is None else bs[4])

    def numerical(self, sm, sp, nrm):
        """Inviscid numerical flux . n and the two sides' F . n."""
        fm = (self.inviscid(sm) * nrm[None]).sum(1)
        fp = (self.inviscid(sp) * nrm[None]).sum(1)
        um, up = (sm["v"] * nrm).sum(0), (sp["v"] * nrm).sum(0)
        if self.case["flux"] == "rusanov":
            lam = torch.maximum((sm["v"] ** 2).sum(0).sqrt() + sm["c"],
                                (sp["v"] ** 2).sum(0).sqrt() + sp["c"])
            return 0.5 * (fm + fp + lam * (sm["q"] - sp["q"]))
        ps = 0.5 * (sm["p"] + sp["p"]) + (um - up) * (sm["rho"] + sp["rho"]) * (
            sm["c"] + sp["c"]) / 8
        root = []
        for s in (sm, sp):
            k = 1 + (s["gamma"] + 1) / (2 * s["gamma"]) * (ps / s["p"] - 1)
            root.append(torch.where(ps > s["p"], k, torch.ones_like(k)).sqrt())
        lo, hi = um - sm["c"] * root[0], up + sp["c"] * root[1]
        f = (hi * fm - lo * fp + hi * lo * (sp["q"] - sm["q"])) / (hi - lo)
        return torch.where(lo >= 0, fm, torch.where(hi <= 0, fp, f))

    def rhs(self, q, time=0.0, viscous=True):
        """(right-hand side with the mixture's sources, gradients, T)."""
        d = self.dim
        t = self.temperature(q, None if not torch.is_tensor(self.tseed) else
                             self.tseed.to(self.dev))
        bs = self.boundary_states(q, t, time)
        s = self.state(q, t)
        flux = -self.inviscid(s)
        gq = gt = fv = None
        if viscous:
            gq, gt = self.gradients(q, t, bs)
            fv = self.viscous(s, gq, gt)
            flux = flux + fv
        nrm = self.nrm.permute(2, 0, 1)[..., None]
        nb = None if bs is None else bs[0]
        sm = self.state(self.inside(q), self.inside(t))
        sp = self.state(self.outside(q, nb), self.outside(t, None if bs is None else bs[1]))
        star = -self.numerical(sm, sp, nrm.expand(sm["v"].shape))
        if viscous:
            fb = None
            if bs is not None:
                bm = self.viscous(self.state(self.at_boundary(q), self.at_boundary(t)),
                                  self.at_boundary(gq), self.at_boundary(gt))
                fb = 2 * self.viscous_at_walls(q, bs, gq, gt) - bm
            star = star + 0.5 * ((self.inside(fv) + self.outside(fv, fb)) * nrm[None]).sum(1)
        out = []
        for c in range(q.shape[0]):
            g = torch.einsum("erj,jek->rek", self.rx, flux[c])
            out.append(self.lifted(star[c]) - torch.einsum("rik,rek->ei", self.weak, g))
        out = torch.stack(out)
        if self.mix:
            out[2 + d:] += self.sources(q, t)
        return out, gq, gt, t

    def viscous_at_walls(self, q, bs, gq, gt):
        """F_V of the boundary states with the walls' gradients."""
        d = self.dim
        qm, gqm, gtm = self.at_boundary(q), self.at_boundary(gq), self.at_boundary(gt)
        n = self.nrm[self.be, self.bf].T[:, :, None]
        wall = (self.side >= 2)[:, None].expand_as(qm[0])
        adiabatic = (self.side >= 4)[:, None].expand_as(qm[0])
        y = qm[2 + d:] / qm[0]
        gy = (gqm[2 + d:] - y[:, None] * gqm[0]) / qm[0]
        gy = gy - (gy * n[None]).sum(1, keepdim=True) * n[None]
        gqb = gqm.clone()
        gqb[2 + d:] = torch.where(wall, qm[0] * gy + y[:, None] * gqm[0], gqm[2 + d:])
        gtb = torch.where(adiabatic, gtm - (gtm * n).sum(0) * n, gtm)
        return self.viscous(self.state(bs[2], bs[3]), gqb, gtb)


def _exact_train(case, seed):
    net, x, target = _train_inputs(case, seed)
    p = net.params.double().requires_grad_(True)
    o, parts = 0, []
    for shape in ((H, KIN), (H,), (H, H), (H,), (H,), (1,)):
        n = math.prod(shape)
        parts.append(p[o:o + n].reshape(shape))
        o += n
    w1, b1, w2, b2, w3, b3 = parts
    h = torch.tanh(x.double() @ w1[:, :8].T + b1)
    h = torch.tanh(h @ w2.T + b2)
    loss = ((h @ w3 + b3 - target.double()) ** 2).mean()
    loss.backward()
    g, k = p.grad, net.step_count + 1
    m = BETA1 * net.m.double() + (1 - BETA1) * g
    v = BETA2 * net.v.double() + (1 - BETA2) * g * g
    new = p.detach() - LR * (m / (1 - BETA1 ** k)) / ((v / (1 - BETA2 ** k)).sqrt() + EPS)
    pad = torch.zeros((H, KIN), dtype=torch.bool, device=new.device)
    pad[:, 8:] = True
    new[:H * KIN] = torch.where(pad.ravel(), torch.zeros_like(new[:H * KIN]), new[:H * KIN])
    return dict(loss=loss.detach().reshape(1), grad=g, params=new)


def exact(case, seed):
    if case["call"] == "train":
        return _exact_train(case, seed)
    if work(case)["bytes"] > 1.5e9:
        return None            # minutes of set-up and tens of GB of face arrays
    ex = _Exact(case, seed)
    call = case["call"]
    if call == "temperature":
        return dict(temperature=ex.temperature(ex.q))
    if call == "ns":
        rhs, _, _, t = ex.rhs(ex.q)
        return dict(rhs=rhs, temperature=t) if ex.mix else dict(rhs=rhs)
    if call == "ns_gradients":
        rhs, gq, gt, t = ex.rhs(ex.q)
        return dict(rhs=rhs, grad_cv=gq, grad_t=gt, temperature=t)
    viscous = call != "euler_step"
    dt = DT_REACTING if viscous else DT_VORTEX

    def f(t, q):
        return ex.rhs(q, t, viscous)[0]
    q = ex.q
    k1 = f(0.0, q)
    k2 = f(dt / 2, q + dt / 2 * k1)
    k3 = f(dt / 2, q + dt / 2 * k2)
    k4 = f(dt, q + dt * k3)
    new = q + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    return dict(state=new, state32=new) if call == "reacting_step" else dict(state=new)

# }}}
