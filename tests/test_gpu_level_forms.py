"""The coarse-level products of the Standard V-cycle in each of their forms against a matrix-free restatement of the
cycle in numpy, which knows no coarse element matrices: A_1 = M P^T M K(E) M P M is applied through the finest grid,
P the Kronecker product of the three linear interpolations.  Spans of 2 only (mg_nondyadic = 0) and three levels, so
that level 1 has 11,781 nodes (split form), 25,725 (a thread per node or row, on a ragged grid) and 61,161 (FP32:
unrolled); none is a multiple of a block's nodes.  The coarsest level is solved by Jacobi (more than 1000 DOFs).
Then the forms in one batch: members with each of them equal their solo runs bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

CORNER_D = [(0, 1, 0), (1, 1, 0), (1, 0, 0), (0, 0, 0), (0, 1, 1), (1, 1, 1), (1, 0, 1), (0, 0, 1)]


def interpolation(nf, s):
    i = np.arange(nf + 1)
    c = np.minimum(i // s, nf // s - 1)
    t = (i - c * s) / s
    return sp.csr_matrix((np.concatenate([1 - t, t]), (np.tile(i, 2), np.concatenate([c, c + 1]))),
                         shape=(nf + 1, nf // s + 1))


class Restatement:
    def __init__(self, P, E, w=float(np.float32(0.35))):   # t3d_params.mg_standard_weight is a float
        self.w, (nx, ny, nz), self.Ke, self.E = w, P.res, P.ke(), E
        cz, rem = np.divmod(P.ele_map_back().astype(np.int64), nx * ny)
        cx, cy = np.divmod(rem, ny)
        n = np.stack([((cz + dz) * (ny + 1) + cy + dy) * (nx + 1) + cx + dx for dx, dy, dz in CORNER_D], axis=1)
        self.dofs = (3 * n[:, :, None] + np.arange(3)).reshape(-1, 24)
        self.M = [(P.mg_mask(l) == 0).astype(float) for l in range(3)]
        self.D = [P.mg_diag(l) for l in range(3)]
        self.P = [None]
        for l in (1, 2):
            fx, fy, fz = P.levels[l - 1][:3]
            s = P.levels[l][3]
            nodes = sp.kron(interpolation(fz, s), sp.kron(interpolation(fy, s), interpolation(fx, s)))
            self.P.append(sp.kron(nodes, sp.identity(3)).tocsr())

    def A(self, l, x):
        x = self.M[l] * x
        if l == 0:
            f = (x[self.dofs] @ self.Ke) * self.E[:, None]
            y = np.bincount(self.dofs.ravel(), f.ravel(), x.size)
        else:
            y = self.P[1].T @ self.A(0, self.P[1] @ x)
        return self.M[l] * y

    def apply(self, r0):
        r, x = [r0, None, None], [None] * 3
        for l in (0, 1):
            x[l] = self.M[l] * (self.w * r[l] / self.D[l])
            r[l + 1] = self.M[l + 1] * (self.P[l + 1].T @ (self.M[l] * (r[l] - self.A(l, x[l]))))
        x[2] = self.M[2] * r[2] / self.D[2]
        for l in (1, 0):
            x[l] = self.M[l] * (x[l] + self.P[l + 1] @ x[l + 1])
            x[l] = self.M[l] * (x[l] + self.w * (r[l] - self.A(l, x[l])) / self.D[l])
        return x[0]


@pytest.mark.parametrize("dims, nodes", [((32, 64, 40), 11781), ((39, 95, 47), 25725), ((56, 112, 72), 61161)])
def test_level_product_forms_match_restatement(dims, nodes):
    import algorithmengineering_altproject_b200 as t3d
    P = t3d.Problem(*dims, mg_vcycle=t3d.T3D_VCYCLE_STANDARD, precision=t3d.T3D_MIXED, mg_nondyadic=0, mg_max_levels=3)
    assert P.coarse_n == 0 and np.prod([v + 1 for v in P.levels[1][:3]]) == nodes
    rng = np.random.default_rng(41)
    E = rng.uniform(1e-3, 1.0, P.ne)
    P.make_diagonal_preconditioner_from_static(E)
    R = Restatement(P, E)
    fd = P.free_dofs().astype(np.int64)
    rf = rng.standard_normal(P.nf).astype(np.float32).astype(np.float64)
    r = np.zeros(R.M[0].size)
    r[fd] = rf
    ref = R.apply(r)[fd]
    assert np.linalg.norm(P.vcycle(rf) - ref) <= 1e-10 * np.linalg.norm(ref)
    assert np.linalg.norm(P.vcycle32(rf) - ref) <= 1e-5 * np.linalg.norm(ref)
    P.close()


def test_batch_of_all_forms_equals_solo():
    import algorithmengineering_altproject_b200 as t3d
    regime = dict(oc_sum_order=1, mg_coarse_assembly=1, mg_vcycle=1, mg_rebuild_period=1, cg_tol=1e-6, cg_max_it=2000)
    dims, V0 = [(128, 256, 128), (96, 192, 96), (16, 48, 24)], [0.12, 0.1, 0.2]   # level 1: 70,785, 30,625 and 175 nodes
    B = t3d.Batch(dims, **regime)
    cs = B.design_init(V0)
    recs = B.run([1, 1, 1])
    xs = [m.density() for m in B.members]
    B.close()
    for i, d in enumerate(dims):
        P = t3d.Problem(*d, precision=t3d.T3D_MIXED, matvec32_tile=t3d.T3D_BATCH_TILE, **regime)
        assert P.design_init(V0[i]) == cs[i]
        r = P.design_step()
        assert (r["obj"], r["pcg_iters"]) == (recs[i][0]["obj"], recs[i][0]["pcg_iters"])
        np.testing.assert_array_equal(P.density(), xs[i])
        P.close()
