"""Elements whose directions differ by orders of magnitude, far from the origin
or in nearly still fluid: fixed-point sums have a unit where FP64 sums have one
per value, so each field and each variable is compared with extended precision
by itself, against what plain FP64 is off."""
import numpy as np
import pytest

import cases
from oracle.oracle import ExtendedOracle, Oracle

pytestmark = pytest.mark.gpu

M, R, S = cases.M, cases.R, cases.S
LD = np.longdouble


def _mesh(basis, shape, p, cells, lengths, offset=0.0):
    ra = R.reference_approximation(basis, shape, p, mapping_degree=p)
    limits = tuple((offset if m == 0 else 0.0, (offset if m == 0 else 0.0) + L) for m, L in enumerate(lengths))
    mesh = M.uniform_periodic_mesh(ra, limits, (cells,) * len(lengths))
    return ra, M.warp_mesh(mesh, ra, "Chan", 0.05, tuple(lengths))


def _extended_factors(mesh, ra, metrics):
    """Geometric factors of a tetrahedral mesh in long double, by component."""
    ext = lambda a: [np.asarray(v).astype(LD) for v in a]  # noqa: E731
    mo = M.metric_operators(ra, metrics, True)
    x, D, n = ext(mesh.xyz), ext(mo.Drst), ext(mo.nrstJ)
    if metrics == "Exact":
        def at(T):
            T = T.astype(LD)
            a = np.stack([np.stack([(x[m] @ D[k].T) @ T.T for k in range(3)], -1) for m in range(3)], -2)
            J, A = M._adjugate_3(a)
            return J, A.transpose(0, 3, 2, 1)
        (Jq, Lq), (_, Lf) = at(mo.Vq), at(mo.Vf)
        Jq = Jq @ mo.project.astype(LD).T
    else:
        d = [[v @ Dm.T for Dm in D] for v in x]
        J = (d[0][0] * (d[1][1] * d[2][2] - d[2][1] * d[1][2]) - d[1][0] * (d[0][1] * d[2][2] - d[2][1] * d[0][2])
             + d[2][0] * (d[0][1] * d[1][2] - d[1][1] * d[0][2]))
        Jq = J @ mo.Vq.astype(LD).T
        t = M._curl_metrics_3d(*[v @ mo.N_to_N1.astype(LD).T for v in x], *ext(mo.D1))
        Lq, Lf = [np.stack([np.stack([t[3 * a + b] @ T.astype(LD).T for b in range(3)], 1) for a in range(3)], 1)
                  for T in (mo.Vq1, mo.Vf1)]
    nJf = np.stack([sum(Lf[:, a, m] * n[m] for m in range(3)) for a in range(3)], -1)
    out = {"J_q": Jq, "J_f": np.sqrt((nJf * nJf).sum(-1))}
    out.update({("Lambda_q", a, b): Lq[:, a, b] for a in range(3) for b in range(3)})
    out.update({("nJf", a): nJf[..., a] for a in range(3)})
    return out


def _component(gf, key):
    if isinstance(key, str):
        return getattr(gf, key)
    return gf.nJf[..., key[1]] if key[0] == "nJf" else gf.Lambda_q[:, key[1], key[2]]


@pytest.mark.parametrize("metrics", ["ChanWilcox", "Exact"])
@pytest.mark.parametrize("p", [2, 4])
@pytest.mark.parametrize("aspect,offset", [(1.0, 0.0), (1.0, 1.0e3), (1.0e2, 0.0), (1.0e4, 0.0), (1.0e6, 0.0),
                                           (1.0e4, 1.0e4)])
def test_geometric_factors(gpu_lib, pkg, metrics, p, aspect, offset):
    """Every component of the factors of a box 1 : 1 : 1/aspect at an offset
    along x: no further from long double than twice the host's FP64 evaluation,
    and a few units in the last place (two evaluations of one sum differ by
    about their own errors)."""
    ra, mesh = _mesh("ModalTensor", "Tet", p, 2, (2 * np.pi, 2 * np.pi, 2 * np.pi / aspect), offset)
    want = _extended_factors(mesh, ra, metrics)
    got = pkg.gb300.geometric_factors(mesh, ra, metrics, True)
    host = M.spatial_discretization(mesh, ra, metrics=metrics).geometric_factors
    for key, w in want.items():
        scale = np.abs(w).max()
        err, err64 = [float(np.abs(_component(gf, key) - w).max() / scale) for gf in (got, host)]
        assert err <= 2.0 * err64 + 4.0 * 2.0 ** -52, (key, err, err64)


class _Shear:
    """Smooth density and pressure, every velocity component ``speed[m]`` times a
    periodic function of two coordinates."""

    def __init__(self, lengths, speed):
        self.k, self.speed = [2 * np.pi / L for L in lengths], speed

    def evaluate(self, x, t=0.0):
        k, d = self.k, len(self.k)
        rho = 1.0 + 0.05 * np.sin(k[0] * x[0] + 0.3) * np.cos(k[-1] * x[-1])
        p = (1.0 + 0.05 * np.cos(k[-1] * x[-1])) / 1.4
        v = [self.speed[m] * np.cos(k[m] * x[m] + 0.5 * m) * np.sin(k[(m + 1) % d] * x[(m + 1) % d] + 0.7)
             for m in range(d)]
        E = p / 0.4 + 0.5 * rho * sum(w * w for w in v)
        return np.stack([rho, *[rho * w for w in v], E], axis=-1)


def _check_variables(basis, shape, p, lengths, speed, ec):
    """Every variable of the residual no further from extended precision than
    four times the FP64 oracle (as the residuals of other flows are held to)."""
    ra, mesh = _mesh(basis, shape, p, 1 if shape == "Tet" else 2, lengths)
    sd = M.spatial_discretization(mesh, ra, metrics="ChanWilcox")
    nflux = S.EntropyConservativeNumericalFlux() if ec else S.LaxFriedrichsNumericalFlux()
    host = S.HostArrays(S.EulerEquations(len(lengths), 1.4), sd, S.FluxDifferencingForm(inviscid_numerical_flux=nflux))
    u = S.initialize(_Shear(lengths, speed), sd)
    got, want = cases.PKG.GB300Solver(host).residual(u), ExtendedOracle(host).residual(u)
    fp64 = [Oracle(host).residual(u), Oracle(host, variant="fma").residual(u)]
    for e in range(host.N_c):
        err, err64 = [max(float(np.linalg.norm(r[:, e] - want[:, e])) for r in rs) for rs in ([got], fp64)]
        assert err <= 4.0 * err64 + 1.0e-14 * np.linalg.norm(want[:, e]), (e, err / err64)


@pytest.mark.parametrize("basis,shape,p", [("ModalTensor", "Tri", 3), ("NodalTensor", "Tri", 4), ("ModalTensor", "Tet", 2),
                                           ("ModalTensor", "Tet", 4), ("NodalTensor", "Tet", 3)])
@pytest.mark.parametrize("aspect", [7.0, 9.0, 1.0e2, 1.0e4])
@pytest.mark.parametrize("along", ["long", "short"])
@pytest.mark.parametrize("ec", [True, False])
def test_residual(gpu_lib, basis, shape, p, aspect, along, ec):
    """Boxes with one short side, on both sides of the fixed-point terms' limit
    and far beyond it, with flow along the long sides or across them."""
    d = 2 if shape == "Tri" else 3
    long, short = (0.3, 0.3 / aspect) if along == "long" else (0.3 / aspect, 0.3)
    _check_variables(basis, shape, p, (2 * np.pi,) * (d - 1) + (2 * np.pi / aspect,), (long,) * (d - 1) + (short,), ec)


@pytest.mark.parametrize("basis,shape,p", [("ModalTensor", "Tri", 4), ("NodalTensor", "Tet", 3)])
@pytest.mark.parametrize("mach", [1.0e-6, 1.0e-7, 1.0e-9, 1.0e-12])
def test_low_mach_without_dissipation(gpu_lib, basis, shape, p, mach):
    """Velocities next to and below the smallest fixed-point unit, where no
    Lax-Friedrichs term hides what they lose."""
    d = 2 if shape == "Tri" else 3
    _check_variables(basis, shape, p, (2 * np.pi,) * d, (mach,) * d, True)
