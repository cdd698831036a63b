"""Fixed-point operators of the FP64 form with caller-supplied operators and
geometry that the built-in rules do not produce."""
import numpy as np
import pytest

import cases
from oracle.oracle import ExtendedOracle, Oracle, rel2

pytestmark = pytest.mark.gpu

S = cases.S


def _problem(shape, p):
    """Host arrays and a smooth subsonic state, both the caller's to change."""
    d = 2 if shape == "Tri" else 3
    sd = cases._disc("ModalTensor", shape, p, 3 if d == 2 else 1, 2 * np.pi, 0.05, "ChanWilcox")
    host = S.HostArrays(S.EulerEquations(d, 1.4), sd,
                        S.FluxDifferencingForm(inviscid_numerical_flux=S.LaxFriedrichsNumericalFlux()))

    class Flow:
        def evaluate(self, x, t=0.0):
            rho = 1.0 + 0.05 * np.sin(x[0] + 0.3)
            v = [0.4 * np.cos(x[m] + 0.5 * m) for m in range(d)]
            E = (1.0 + 0.05 * np.cos(x[-1])) / 1.4 / 0.4 + 0.5 * rho * sum(w * w for w in v)
            return np.stack([rho, *[rho * w for w in v], E], axis=-1)

    return host, S.initialize(Flow(), sd)


@pytest.mark.parametrize("shape,p", [("Tri", 3), ("Tet", 2)])
def test_selection_rows_of_the_facet_interpolation(gpu_lib, shape, p):
    """Rows of R that pick one volume node, with a weight next to one (volume
    nodes on the facets): the nodal values are those of the nodes, to the parity
    tolerance of 1e-12, and the residual is no further from extended precision
    than four times the FP64 oracle."""
    host, u = _problem(shape, p)
    rows, val = host.R.rowval - 1, host.R.nzval
    for j in range(host.N_f):
        mine = np.flatnonzero(rows == j)
        keep = mine[np.argmax(np.abs(val[mine]))]
        val[mine] = 0.0
        val[keep] = np.nextafter(1.0, 0.0)
    gpu = cases.PKG.GB300Solver(host)
    got_q, got_f = gpu.nodal_values(u)
    want_q, want_f = Oracle(host).nodal_values(u)
    assert rel2(got_q, want_q) <= 1.0e-12 and rel2(got_f, want_f) <= 1.0e-12
    want = ExtendedOracle(host).residual(u)
    e64 = max(rel2(Oracle(host).residual(u), want), rel2(Oracle(host, variant="fma").residual(u), want))
    assert rel2(gpu.residual(u), want) <= 4.0 * e64 + 1.0e-14


@pytest.mark.parametrize("field,value", [("JinvW", np.nan), ("JinvW", np.inf), ("WJ", np.nan), ("WJ", np.inf), ("J", 0.0)])
def test_non_finite_geometry_is_reported(gpu_lib, field, value):
    """One weight or mass entry of one element that is not finite, or a Jacobian
    of zero, ends in SSE_ERR_NONPHYSICAL and not in numbers."""
    host, u = _problem("Tet", 2)
    if field == "J":
        host.WJ[-1, 3], host.JinvW[-1, 3] = 0.0, np.inf
    else:
        getattr(host, field)[-1, 3] = value
    with pytest.raises(cases.PKG.SSEError) as err:
        cases.PKG.GB300Solver(host).residual(u)
    assert err.value.code == cases.PKG.abi.SSE_ERR_NONPHYSICAL


@pytest.mark.parametrize("unit", [1.0e-45, 1.0e45])
def test_lengths_in_other_units(gpu_lib, unit):
    """The same mesh with lengths of 1e-45 and 1e45: Jacobians of 1e-135 and 1e135
    lie beyond the exponents of the scaled mass operators.  The residual is that
    of unit lengths over the unit, to the parity tolerance of 1e-12."""
    host, u = _problem("Tet", 2)
    want = cases.PKG.GB300Solver(host).residual(u) / unit
    for name, power in (("WJ", 3), ("JinvW", -3), ("BJf", 2), ("Lambda_q", 2), ("halfnJf", 2), ("halfnJq", 2)):
        getattr(host, name)[...] *= unit ** power
    assert rel2(cases.PKG.GB300Solver(host).residual(u) * unit, want * unit) <= 1.0e-12
