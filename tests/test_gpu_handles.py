"""Several handles of one process: a new handle leaves those before it as they
were."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

S, setups = cases.S, cases.setups


def _problem(p, form):
    pb = setups.tgv_tet(cells=1, p=p)
    forms = {"fixed point": pb.form,
             "fp64": S.FluxDifferencingForm(inviscid_numerical_flux=S.LaxFriedrichsNumericalFlux(),
                                            two_point_flux=S.ChandrashekarFlux()),
             "standard": S.StandardForm(inviscid_numerical_flux=S.LaxFriedrichsNumericalFlux())}
    return S.HostArrays(pb.law, pb.sd, forms.get(form, pb.form)), pb.u0


@pytest.mark.parametrize("form", ["fixed point", "fp64", "standard", "mixed", "transpose"])
def test_smaller_handle_after_a_larger(gpu_lib, form):
    """Kernels of any element size are shared by the handles; the larger element
    still has its shared memory after a handle for a smaller one, bit for bit."""
    big, u = _problem(6 if form in ("fixed point", "fp64") else 5, form)
    small, _ = _problem(1, form)

    def solver(host):
        s = cases.PKG.GB300Solver(host)
        if form == "mixed":
            s.set_precision(cases.PKG.abi.SSE_MIXED)
        return s

    def run(s, v):
        return s.residual_vjp(v, np.cos(np.arange(v.size)).reshape(v.shape)) if form == "transpose" else s.residual(v)

    first = solver(big)
    want = run(first, u)
    second = solver(small)
    run(second, _problem(1, form)[1])
    assert np.array_equal(run(first, u), want)
