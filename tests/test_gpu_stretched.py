"""Elements whose directions differ by orders of magnitude, far from the origin
or in nearly still fluid: fixed-point sums have a unit where FP64 sums have one
per value, so each field and each variable is compared with extended precision
by itself, against what plain FP64 is off."""
import numpy as np
import pytest

import cases

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
