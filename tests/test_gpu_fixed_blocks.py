"""Which elements of the FP64 form are evaluated in fixed point: those of every
block without an element out of range, and only those."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

S = cases.S


@pytest.mark.parametrize("shape,p,cells,basis,most", [("Tri", 3, 12, "ModalTensor", 4 * 7), ("Tri", 4, 12, "NodalTensor", 4 * 3),
                                                      ("Tet", 2, 3, "ModalTensor", 5)])
def test_blocks_out_of_range(gpu_lib, shape, p, cells, basis, most):
    """One element's density 200 times its neighbours': it and the elements that
    face it are out of range.  Others see the same data: those in the blocks of
    these (``most`` at most) now come from the FP64 passes and agree to the parity
    tolerance, with bits that show it; the rest keep their bits."""
    d = 2 if shape == "Tri" else 3
    sd = cases._disc(basis, shape, p, cells, 2 * np.pi, 0.05, "ChanWilcox")
    host = S.HostArrays(S.EulerEquations(d, 1.4), sd,
                        S.FluxDifferencingForm(inviscid_numerical_flux=S.LaxFriedrichsNumericalFlux()))

    class Flow:
        def evaluate(self, x, t=0.0):
            rho = 1.0 + 0.05 * np.sin(x[0] + 0.3)
            v = [0.4 * np.cos(x[m] + 0.5 * m) for m in range(d)]
            E = (1.0 + 0.05 * np.cos(x[-1])) / 1.4 / 0.4 + 0.5 * rho * sum(w * w for w in v)
            return np.stack([rho, *[rho * w for w in v], E], axis=-1)

    u = S.initialize(Flow(), sd)
    solver = cases.PKG.GB300Solver(host)
    before = solver.residual(u)
    k = host.N_e // 2
    u[k] *= 200.0
    after = solver.residual(u)
    facing = (np.asarray(host.mapP).reshape(host.N_e, host.N_f)[k] - 1) // host.N_f
    others = np.setdiff1d(np.arange(host.N_e), np.append(facing, k))
    changed = [e for e in others if not np.array_equal(before[e], after[e])]
    assert 0 < len(changed) <= most
    scale = np.abs(before).max(axis=(0, 2))
    for e in changed:
        assert np.all(np.abs(after[e] - before[e]).max(axis=1) <= 1.0e-12 * scale)
