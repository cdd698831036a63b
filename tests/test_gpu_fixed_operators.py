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
