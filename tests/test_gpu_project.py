"""L2 projection of initial data on the GPU (sse_project_function) against
the host restatement of project_function (Solvers.jl:396-418)."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["vortex_tri_modal", "tgv_tet_modal", "tgv_tet_p5", "tgv_tet_p6",
                                  "multi_tri", "multi_tet"])
def test_projection_matches_host(name, gpu_lib, pkg):
    host, _ = cases.make(name)
    sd = host.sd
    if "tet" in name:
        ic = pkg.solver.TaylorGreenVortex(1.4, 0.1)
    else:
        ic = pkg.setups.vortex_tri(cells=2, p=2).initial_data
    want = pkg.solver.initialize(ic, sd)
    got = pkg.solver.initialize(ic, sd, projection="gpu")
    err = np.abs(got - want).max() / np.abs(want).max()
    assert err < 1e-12, err


def test_projection_device_buffers(gpu_lib, pkg):
    import torch
    host, _ = cases.make("tgv_tet_modal")
    sd = host.sd
    ra = sd.reference_approximation
    uq = pkg.solver.TaylorGreenVortex(1.4, 0.1).evaluate(sd.mesh.xyzq, 0.0).transpose(0, 2, 1)
    uq = np.ascontiguousarray(uq)
    a = pkg.gb300.project_function(ra, sd.geometric_factors.J_q, uq)
    b = pkg.gb300.project_function(ra, torch.from_numpy(sd.geometric_factors.J_q).cuda(),
                                   torch.from_numpy(uq).cuda())
    assert np.array_equal(a, b.cpu().numpy())


def test_projection_rejects_a_negative_jacobian(gpu_lib, pkg):
    """A mass matrix that is not positive definite is an error, as the
    reference's cholesky throws."""
    host, _ = cases.make("vortex_tri_modal")
    sd = host.sd
    J = sd.geometric_factors.J_q.copy()
    J[3] *= -1.0
    uq = np.ones((sd.N_e, 4, J.shape[1]))
    with pytest.raises(pkg.SSEError) as e:
        pkg.gb300.project_function(sd.reference_approximation, J, uq)
    assert e.value.code == pkg.abi.SSE_ERR_NONPHYSICAL


@pytest.mark.parametrize("shape,p", [("Tri", 1), ("Tri", 2), ("Tri", 5), ("Tet", 1), ("Tet", 3), ("Tet", 6)])
@pytest.mark.parametrize("scale", [1.0, 3.0e-40, 7.0e30])
def test_sizes_and_units(gpu_lib, pkg, shape, p, scale):
    """Tiles of M that np does not fill, node counts that are no multiple of
    four, and data far from one: within 1e-12 of each projection's largest
    coefficient (as test_projection's whole-vector bound), and an element of zero
    data stays zero."""
    d = 2 if shape == "Tri" else 3
    ra = cases.R.reference_approximation("ModalTensor", shape, p, mapping_degree=p)
    mesh = cases.M.uniform_periodic_mesh(ra, ((0.0, 1.0),) * d, (2,) * d)
    J = cases.M.spatial_discretization(mesh, ra, metrics="Exact").geometric_factors.J_q
    uq = scale * (1.0 + np.stack([np.sin(x) for x in mesh.xyzq], axis=1))
    uq[0] = 0.0
    got = pkg.gb300.project_function(ra, J, np.ascontiguousarray(uq))
    V, WJ = ra.V, ra.W[None, :] * J
    mass = np.einsum("qa,kq,qb->kab", V, WJ, V)
    want = np.linalg.solve(mass, np.einsum("qa,keq->kae", V, uq * WJ[:, None, :])).transpose(0, 2, 1)
    assert np.all(got[0] == 0.0)
    assert np.abs(got - want).max() <= 1.0e-12 * np.abs(want).max()


@pytest.mark.parametrize("N_p,N_q,N_c,N_e", [(1, 1, 1, 1), (10, 16, 4, 5), (35, 125, 5, 7), (84, 343, 5, 3), (120, 120, 8, 3),
                                             (165, 166, 1, 2), (168, 168, 1, 2)])
def test_partial_blocks_chunks_and_large_elements(gpu_lib, pkg, N_p, N_q, N_c, N_e):
    """Element counts that do not fill a block, nodes that do not fill a chunk,
    and elements whose mass matrix leaves shared memory for a part of a chunk or
    none.  VDM has orthonormal columns and W J lies in [1/2, 3/2], so the mass
    matrix has a condition of at most 3 and sums of N_q terms stay within
    1e-12."""
    rng = np.random.default_rng([N_p, N_q])

    class Approximation:
        V = np.linalg.qr(rng.standard_normal((N_q, N_p)))[0]
        W = np.ones(N_q)

    J = rng.uniform(0.5, 1.5, (N_e, N_q))
    uq = rng.standard_normal((N_e, N_c, N_q))
    got = pkg.gb300.project_function(Approximation, J, uq)
    V = Approximation.V
    mass = np.einsum("qa,kq,qb->kab", V, J, V)
    want = np.linalg.solve(mass, np.einsum("qa,keq->kae", V, uq * J[:, None, :])).transpose(0, 2, 1)
    assert np.abs(got - want).max() <= 1.0e-12 * np.abs(want).max()
