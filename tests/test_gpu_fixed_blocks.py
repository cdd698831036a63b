"""Which elements of the FP64 form are evaluated in fixed point: those of every
block without an element out of range, and only those."""
import numpy as np
import pytest

import cases
from oracle.oracle import Oracle, rel2

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


def _phases(basis="ModalTensor", shape="Tet", aspect=1.0, form=None, law=None, multi=False):
    d = 2 if shape == "Tri" else 3
    if multi:
        sd = cases._disc_multi(basis, shape, 3, 2, 2 * np.pi, 0.05, "ChanWilcox")
    else:
        ra = cases.R.reference_approximation(basis, shape, 3, mapping_degree=3)
        box = (2 * np.pi,) * (d - 1) + (2 * np.pi / aspect,)
        mesh = cases.M.uniform_periodic_mesh(ra, tuple((0.0, L) for L in box), (2,) * d)
        sd = cases.M.spatial_discretization(cases.M.warp_mesh(mesh, ra, "Chan", 0.05, box), ra, metrics="ChanWilcox")
    form = form or S.FluxDifferencingForm(inviscid_numerical_flux=S.LaxFriedrichsNumericalFlux())
    return cases.PKG.GB300Solver(S.HostArrays(law or S.EulerEquations(d, 1.4), sd, form)).fixed_point_phases()


def test_reported_phases(gpu_lib):
    """What a handle says of its phases: A needs a modal tensor-product basis, B the
    entropy-conservative flux, gamma of at most 1.7 and elements not stretched."""
    A, B = cases.PKG.abi.SSE_FIXED_POINT_A, cases.PKG.abi.SSE_FIXED_POINT_B
    lf = S.LaxFriedrichsNumericalFlux()
    assert _phases() == _phases(shape="Tri") == A + B
    assert _phases("NodalTensor") == _phases("ModalMulti", multi=True) == B
    assert _phases(aspect=1.0e3) == A
    assert _phases(law=S.EulerEquations(3, 2.0)) == 0
    assert _phases(form=S.StandardForm(inviscid_numerical_flux=lf)) == 0
    assert _phases(form=S.FluxDifferencingForm(inviscid_numerical_flux=lf, two_point_flux=S.ChandrashekarFlux())) == 0


@pytest.mark.parametrize("shape,p,fp64,fixed", [("Tri", 1, 38, 39), ("Tri", 2, 28, 29), ("Tri", 7, 13, 14), ("Tet", 1, 5, 6),
                                                ("Tri", 3, None, 2), ("Tet", 2, None, 1)])
def test_size_where_phase_a_turns_to_fixed_point(gpu_lib, shape, p, fp64, fixed):
    """The meshes (cells a side) on both sides of the line, or the smallest where
    there is none: the phase that runs, and its nodal values to the parity
    tolerance."""
    d = 2 if shape == "Tri" else 3
    for cells, want in ((fp64, 0), (fixed, cases.PKG.abi.SSE_FIXED_POINT_A)):
        if cells is None:
            continue
        sd = cases._disc("ModalTensor", shape, p, cells, 2 * np.pi, 0.05, "ChanWilcox")
        host = S.HostArrays(S.EulerEquations(d, 1.4), sd,
                            S.FluxDifferencingForm(inviscid_numerical_flux=S.LaxFriedrichsNumericalFlux()))
        rng = np.random.default_rng(cells)
        u = np.zeros((host.N_e, host.N_c, host.N_p))
        u[:, 0, 0], u[:, 1, 0], u[:, -1, 0] = 1.0, 0.3, 2.5
        u += 1.0e-3 * rng.standard_normal(u.shape)
        solver = cases.PKG.GB300Solver(host)
        assert solver.fixed_point_phases() & cases.PKG.abi.SSE_FIXED_POINT_A == want
        for got, ref in zip(solver.nodal_values(u), Oracle(host).nodal_values(u)):
            assert rel2(got, ref) <= 1.0e-12
