"""Fixed-point phase B against the oracle where its scales, branches and team
shapes change: jumps on both sides of the means' series branch, elements whose
range sends their block to the FP64 passes (alone and next to others), fluid at
rest, supersonic and low-Mach flow, gamma on both sides of its limit, partial
blocks and every team width (16, 32, 128 and 256 threads, one chunk of pairs
and several)."""
import numpy as np
import pytest

import cases
from oracle.oracle import ExtendedOracle, Oracle, rel2

pytestmark = pytest.mark.gpu

S, setups = cases.S, cases.setups

# (element, degree, cells, basis): 16-, 32-, 128- and 256-thread teams
SHAPES = [("Tri", 2, 3, "ModalTensor"), ("Tri", 4, 5, "NodalTensor"), ("Tet", 2, 1, "ModalTensor"),
          ("Tet", 3, 1, "NodalTensor"), ("Tet", 4, 1, "ModalTensor"), ("Tet", 5, 1, "ModalTensor")]


def _host(shape, p, cells, basis, gamma=1.4, ec=False):
    d = 2 if shape == "Tri" else 3
    sd = cases._disc(basis, shape, p, cells, 2 * np.pi, 0.05, "ChanWilcox")
    nflux = S.EntropyConservativeNumericalFlux() if ec else S.LaxFriedrichsNumericalFlux()
    return S.HostArrays(S.EulerEquations(d, gamma), sd, S.FluxDifferencingForm(inviscid_numerical_flux=nflux))


class _Flow:
    """rho and p vary by (1 + jump sin) over several mesh lengths (with a jump
    across the periodic boundary), the velocity has the Mach number ``mach``."""

    def __init__(self, d, gamma, mach, jump):
        self.d, self.gamma, self.mach, self.jump = d, gamma, mach, jump

    def evaluate(self, x, t=0.0):
        rho = 1.0 + self.jump * np.sin(0.2 * x[0] + 0.3)
        p = (1.0 + self.jump * np.cos(0.2 * x[-1])) / self.gamma
        v = [self.mach * np.cos(0.2 * x[m] + 0.5 * m) for m in range(self.d)]
        E = p / (self.gamma - 1.0) + 0.5 * rho * sum(w * w for w in v)
        return np.stack([rho, *[rho * w for w in v], E], axis=-1)


def _check(host, u):
    """No further from the extended-precision residual than four times the FP64
    oracle is (the residual of a nearly uniform flow is a small difference of
    its fluxes, which no FP64 evaluation resolves to 1e-12)."""
    got = cases.PKG.GB300Solver(host).residual(u)
    want = ExtendedOracle(host).residual(u)
    e64 = max(rel2(Oracle(host).residual(u), want), rel2(Oracle(host, variant="fma").residual(u), want))
    assert rel2(got, want) <= 4.0 * e64 + 1.0e-14


@pytest.mark.parametrize("shape,p,cells,basis", SHAPES)
@pytest.mark.parametrize("mach,jump", [(0.0, 1e-3), (1e-4, 1e-2), (0.3, 0.05), (3.0, 0.3)])
def test_against_oracle(gpu_lib, shape, p, cells, basis, mach, jump):
    host = _host(shape, p, cells, basis, ec=mach == 0.3)
    u = S.initialize(_Flow(host.cfg.d, 1.4, mach, jump), host.sd)
    _check(host, u)


@pytest.mark.parametrize("shape,p,cells,basis", SHAPES)
def test_out_of_range_elements_take_fp64(gpu_lib, shape, p, cells, basis):
    """One element with a density 200 times its neighbours': its range, and
    that of the elements facing it, is beyond 2^4; the others stay."""
    host = _host(shape, p, cells, basis)
    u = S.initialize(_Flow(host.cfg.d, 1.4, 0.3, 0.05), host.sd)
    u[host.N_e // 2] *= 200.0
    _check(host, u)


@pytest.mark.parametrize("gamma", [1.1, 5.0 / 3.0, 1.7, 1.75, 2.0])
def test_gamma(gpu_lib, gamma):
    host = _host("Tet", 2, 1, "ModalTensor", gamma=gamma)
    _check(host, S.initialize(_Flow(3, gamma, 0.5, 0.2), host.sd))


def test_fluid_at_rest_stays_at_rest(gpu_lib):
    """Zero velocity: the mass and energy fluxes are exactly zero."""
    host = _host("Tet", 3, 1, "NodalTensor", ec=True)
    u = S.initialize(_Flow(3, 1.4, 0.0, 0.2), host.sd)
    r = cases.PKG.GB300Solver(host).residual(u)
    assert np.all(r[:, 0] == 0.0) and np.all(r[:, 4] == 0.0)


@pytest.mark.parametrize("shape,p,cells", [("Tri", 1, 3), ("Tri", 7, 2), ("Tri", 8, 2), ("Tet", 1, 1), ("Tet", 3, 1),
                                           ("Tet", 6, 1)])
@pytest.mark.parametrize("a,b", [(1.0, 1.0), (3.0e-9, 2.0e5), (7.0e12, 1.0e-6)])
def test_operators_of_the_projection(gpu_lib, shape, p, cells, a, b):
    """Fixed-point operators of the entropy projection at the smallest and
    largest degrees they take (and p = 8, which keeps FP64), in other units of
    density (a) and velocity (b), with a vanishing momentum component: to the
    parity tolerance of nodal values, 1e-12 of each variable."""
    host = _host(shape, p, cells, "ModalTensor")
    u = S.initialize(_Flow(host.cfg.d, 1.4, 0.4, 0.1), host.sd)
    u[:, 2] = 0.0
    u[:, 0] *= a
    u[:, 1:-1] *= a * b
    u[:, -1] *= a * b * b
    got_q, got_f = cases.PKG.GB300Solver(host).nodal_values(u)
    want_q, want_f = Oracle(host).nodal_values(u)
    speed = np.abs(want_q[:, 1]).max()
    for e in range(host.N_c):
        scale = speed if 0 < e < host.N_c - 1 else np.abs(want_q[:, e]).max()
        assert np.abs(got_q[:, e] - want_q[:, e]).max() <= 1.0e-12 * scale
        assert np.abs(got_f[e] - want_f[e]).max() <= 1.0e-12 * scale


@pytest.mark.parametrize("value", [np.nan, np.inf, -1.0])
@pytest.mark.parametrize("variable", [0, 1, -1])
def test_non_physical_states_are_reported(gpu_lib, value, variable):
    if value == -1.0 and variable == 1:
        pytest.skip("a negative momentum is physical")
    host = _host("Tet", 2, 1, "ModalTensor")
    u = S.initialize(_Flow(3, 1.4, 0.4, 0.1), host.sd)
    u[host.N_e - 1, variable] = value
    with pytest.raises(cases.PKG.SSEError) as err:
        cases.PKG.GB300Solver(host).residual(u)
    assert err.value.code == 4


@pytest.mark.parametrize("p", [3, 4])
def test_errors_have_no_direction(gpu_lib, p):
    """Products are rounded to nearest, not down: over the elements of a mesh
    the errors of each variable and mode have a mean within five standard
    deviations of zero (some 175 means: chance exceeds that once in 10^4)."""
    host = _host("Tet", p, 3, "ModalTensor")
    u = S.initialize(_Flow(3, 1.4, 0.1, 0.02), host.sd)
    u = u + 1e-3 * np.random.default_rng(p).standard_normal(u.shape)
    d = cases.PKG.GB300Solver(host).residual(u) - ExtendedOracle(host).residual(u)
    rms = np.sqrt((d * d).mean(axis=0))
    assert np.all(np.abs(d.mean(axis=0)) <= 5.0 * rms / np.sqrt(len(d)))
