"""The element kernels on meshes whose cells group into fans in every way, against the oracle.

The kernels and the oracle both sum FP64 terms of the same formulas in different orders; with
fewer than 100 terms a node and unit-scale data the results agree to 1e-13 relative, and the bar is
the 1e-11 of the other parity tests."""
import numpy as np
import pytest
from scipy import spatial

from helpers import rel_l2
from oracle import Oracle
from platoanalyze_b200 import capi
from platoanalyze_b200.mesh import box_mesh
from platoanalyze_b200.problem import EllipticProblem, ProblemSpec
from platoanalyze_b200.workloads import splitmix_uniform

pytestmark = pytest.mark.gpu
TOL = 1e-11


def axis_fan(n, closed, twist=0.0):
    """n cells around the edge (0, 1): closed, or open with n + 1 ring nodes; the edge is the longest
    of each cell.  twist moves the ring nodes so that no two cells are alike."""
    m = n if closed else n + 1
    angle = 2 * np.pi * np.arange(m) / (n if closed else n + 3)
    ring = np.stack([np.cos(angle), np.sin(angle), twist * np.sin(3 * angle)], 1)
    x = np.concatenate([[[0, 0, -3.0], [0, 0, 3.0]], ring])
    conn = np.array([[0, 1, 2 + k, 2 + (k + 1) % m] for k in range(n)], np.int32)
    return x, conn


def shuffled_box(nx, ny, nz, seed):
    m = box_mesh(nx, ny, nz, 1.1, 0.8, 0.9)
    rng = np.random.default_rng(seed)
    x = m.coords + rng.uniform(-0.12, 0.12, m.coords.shape) * np.array([1.1 / nx, 0.8 / ny, 0.9 / nz])
    perm = rng.permutation(m.num_nodes).astype(np.int32)
    y = np.empty_like(x)
    y[perm] = x
    conn = perm[m.connectivity][rng.permutation(m.num_cells)]
    return y, np.ascontiguousarray(conn, np.int32)


def delaunay(n, shuffle):
    """About 13 n^3 cells around 2 n^3 jittered lattice points, two to a fan; numbered along the lattice with the
    cells in the order of their first nodes, or at random.  Cells below 2 % of the lattice's volume are left out:
    what is left loses two digits at most in its determinants, far inside the bar."""
    rng = np.random.default_rng(n)
    g = np.stack(np.meshgrid(np.arange(2 * n), np.arange(n), np.arange(n), indexing="ij"), -1).reshape(-1, 3)
    x = (g + rng.uniform(-0.3, 0.3, g.shape)) / n
    conn = spatial.Delaunay(x).simplices
    v = x[conn]
    conn = conn[np.abs(np.linalg.det(v[:, :3] - v[:, 3:])) > 0.02 / n ** 3]
    if not shuffle:
        return x, np.ascontiguousarray(conn[np.argsort(conn.min(1), kind="stable")], np.int32)
    perm = rng.permutation(x.shape[0])
    y = np.empty_like(x)
    y[perm] = x
    return y, np.ascontiguousarray(perm[conn][rng.permutation(conn.shape[0])], np.int32)


MESHES = {
    "one cell": lambda: (np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]]), np.array([[0, 1, 2, 3]], np.int32)),
    "closed fan of 3": lambda: axis_fan(3, True, 0.2),
    "closed fan of 6": lambda: axis_fan(6, True, 0.1),
    "closed fan of 7, one ring node too many": lambda: axis_fan(7, True),
    "open fan of 5": lambda: axis_fan(5, False, 0.1),
    "open fan of 6, one ring node too many": lambda: axis_fan(6, False),
    "32 cells around an edge": lambda: axis_fan(32, True),
    "33 cells around an edge": lambda: axis_fan(33, False, 0.02),
    "90 cells around an edge": lambda: axis_fan(90, True, 0.01),
    "two cells on one edge without a common face": lambda: (
        np.array([[0, 0, -3], [0, 0, 3], [1, 0, 0], [0, 1, 0], [-1, 0, 0], [0, -1, 0.3]], float),
        np.array([[0, 1, 2, 3], [0, 1, 4, 5]], np.int32)),
    "box, tiles of 32 fans": lambda: (lambda m: (m.coords, m.connectivity))(box_mesh(7, 5, 4)),
    "shuffled box, tiles of 32 fans": lambda: shuffled_box(9, 7, 6, 1),
    "shuffled box, tiles of 64 fans": lambda: shuffled_box(40, 33, 30, 2),
    "Delaunay, scalar quantities by cells": lambda: delaunay(18, False),
    "Delaunay, shuffled": lambda: delaunay(18, True),
    "Delaunay, fans of single cells": lambda: delaunay(8, False),
    "box, tiles of 128 fans": lambda: (lambda m: (m.coords, m.connectivity))(box_mesh(51, 39, 39)),
}


def close(a, b):
    a = a.cpu().numpy() if hasattr(a, "cpu") else np.asarray(a)
    assert rel_l2(a, b) <= TOL, rel_l2(a, b)
    assert np.abs(a - b).max() <= TOL * max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("name", MESHES)
def test_element_kernels(name):
    x, conn = MESHES[name]()
    N, C = x.shape[0], conn.shape[0]
    fixed = np.array([0, 1, 5], np.int32)
    spec = ProblemSpec(x, conn, 1.7, 0.28, 3.0, 1e-9, [], fixed, np.zeros(3))
    p, orc = EllipticProblem(spec), Oracle.from_spec(spec)
    z = splitmix_uniform(N, 5, 0.3, 1.0)
    u, lam = np.sin(0.3 * np.arange(3 * N) + 0.2), np.cos(0.7 * np.arange(3 * N))
    zd, ud, ld = p.to_dev(z), p.to_dev(u), p.to_dev(lam)
    close(p.vf_value(ud, zd), orc.vf_value(u, z))
    close(p.sf_gradient_u(ud, zd), orc.sf_gradient_u(u, z))
    dz = orc.sf_gradient_z(u, z)
    close(p.sf_gradient_z(ud, zd), dz)
    close(p.vf_gradient_z_apply(ud, zd, ld, p.to_dev(dz)), orc.matvec_plus(1, 3, orc.vf_gradient_z(u, z), lam, dz.copy()))
    f, g, _ = p.criterion_value_and_gradient(zd, ud)
    fo = orc.sf_value(u, z)
    assert abs(f - fo) <= TOL * abs(fo) and abs(p.sf_value(ud, zd) - fo) <= TOL * abs(fo)
    close(g, orc.criterion_gradient(z, u, self_adjoint=True))
    close(p.criterion_gradient(zd, ud)[0], orc.criterion_gradient(z, u, self_adjoint=True))
    close(np.array([p.volume_value(zd)]), np.array([orc.volume_value(z)]))
    close(p.volume_gradient_z(zd), orc.volume_gradient_z(z))
    # the constrained operator, applied without a matrix: fixed dofs keep their value
    free = u.copy()
    free[fixed] = 0.0
    y = orc.sf_gradient_u(free, z)
    y[fixed] = u[fixed]
    close(p.apply_operator(zd, ud, capi.OPERATOR_MATRIX_FREE), y)
    # results repeat bit for bit
    assert (p.vf_value(ud, zd) == p.vf_value(ud, zd)).all() and p.sf_value(ud, zd) == p.sf_value(ud, zd)
    # one density per cell
    ze, orc = splitmix_uniform(C, 6, 0.3, 1.0), Oracle.from_spec(spec, cell_control=True)
    p.set_control_layout("element")
    zed = p.to_dev(ze)
    close(p.vf_value(ud, zed), orc.vf_value(u, ze))
    close(p.sf_gradient_z(ud, zed), orc.sf_gradient_z(u, ze))
    close(np.array([p.sf_value(ud, zed), p.volume_value(zed)]), np.array([orc.sf_value(u, ze), orc.volume_value(ze)]))


@pytest.mark.parametrize("name", ["Delaunay, scalar quantities by cells", "box, tiles of 128 fans"])
def test_element_control_adds(name):
    """One density per cell: the derivative is added to what is there, by cells and by fans."""
    x, conn = MESHES[name]()
    N, C = x.shape[0], conn.shape[0]
    spec = ProblemSpec(x, conn, 1.7, 0.28, 3.0, 1e-9, [], np.array([0, 1, 5], np.int32), np.zeros(3))
    p, orc = EllipticProblem(spec), Oracle.from_spec(spec, cell_control=True)
    p.set_control_layout("element")
    z = splitmix_uniform(C, 6, 0.3, 1.0)
    u, start = np.sin(0.3 * np.arange(3 * N) + 0.2), np.cos(0.1 * np.arange(C))
    # with lambda = u the product is vol eps(u).C.eps(u) s'(rho), twice the energy's derivative
    want = start + 2.0 * orc.sf_gradient_z(u, z)
    ud = p.to_dev(u)
    close(p.vf_gradient_z_apply(ud, p.to_dev(z), ud, p.to_dev(start)), want)


@pytest.mark.parametrize("name", MESHES)
def test_jacobian_write_out(name):
    """The block CRS Jacobian's shared write-out (nine lanes to a block) on the same meshes: ragged last slices,
    rows without upper blocks, rows beyond the row kernel's range.  Sums over a node's cells: the same bar."""
    x, conn = MESHES[name]()
    spec = ProblemSpec(x, conn, 1.7, 0.28, 3.0, 1e-9, [], np.array([0, 1, 5], np.int32), np.zeros(3))
    p, orc = EllipticProblem(spec), Oracle.from_spec(spec)
    z = splitmix_uniform(x.shape[0], 5, 0.3, 1.0)
    u = np.zeros(3 * x.shape[0])
    close(p.vf_gradient_u(p.to_dev(u), p.to_dev(z)).reshape(-1), np.asarray(orc.vf_gradient_u(u, z)).reshape(-1))
