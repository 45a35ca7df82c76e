"""The cooperative Krylov loops (one launch for many iterations) at the sizes where their split of
the rows changes: one slice, a ragged last slice, 16 to 1 warps per slice, the largest that fits,
and one beyond it, which takes the launch-per-stage loop.

With sampled timings on, a handle runs one launch per stage, so the same handle gives both
results.  Both stop at ||b - A x|| <= 1e-10 ||b|| and are held to the 1e-8 that every solution of this
repository is held to."""
import numpy as np
import pytest

from helpers import rel_l2
from oracle import Oracle
from platoanalyze_b200 import capi
from platoanalyze_b200.mesh import box_mesh
from platoanalyze_b200.problem import EllipticProblem, HelmholtzFilter, ProblemSpec, SolverOptions
from platoanalyze_b200.workloads import cantilever, coarse_grid, method_options, splitmix_uniform

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 2), (7, 3, 2), (20, 10, 10), (26, 12, 12), (30, 16, 16), (40, 20, 20), (50, 26, 26), (60, 30, 30), (70, 33, 33)]


@pytest.mark.parametrize("method", ["plain", "chebyshev", "bf16", "fp16", "fp64-chebyshev", "two-level", "two-level-fp16"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_cooperative_matches_launch_per_stage(size, method):
    if method == "fp16":  # the scaled sweep without a coarse space
        opts = SolverOptions(tolerance=1e-10, max_iterations=200000, precision=capi.PRECISION_MIXED_FP16, chebyshev_degree=8)
    elif method == "fp64-chebyshev":
        opts = SolverOptions(tolerance=1e-10, max_iterations=200000, precision=capi.PRECISION_FP64, chebyshev_degree=1)
    else:
        opts = method_options(method, 1e-10, coarse_grid(*size))
    spec = cantilever(*size, opts)
    z = splitmix_uniform(spec.coords.shape[0], 3, 0.2, 1.0)
    p = EllipticProblem(spec)
    zd = p.to_dev(z)
    u, st = p.solution(zd)
    assert st["converged"] and st["fallback"] == 0 and st["relative_residual"] <= 1e-10, st
    p.set_timing(True)
    v, sv = p.solution(zd)
    assert sv["converged"] and sv["fallback"] == 0
    # (the iteration counts of the one-level flexible methods depend on the last bits of the dot products:
    # the truncated recurrence keeps one direction, so they are not compared)
    if method in ("plain", "two-level", "two-level-fp16"):
        assert abs(st["iterations"] - sv["iterations"]) <= max(3, sv["iterations"] // 20), (st, sv)
    assert rel_l2(u.cpu().numpy(), v.cpu().numpy()) <= 1e-8
    if spec.coords.shape[0] < 4000:
        uo, _, _ = Oracle.from_spec(spec).solution_refined(z, tol=1e-13)
        assert rel_l2(u.cpu().numpy(), uo) <= 1e-8


@pytest.mark.parametrize("method", ["plain", "chebyshev", "two-level"])
def test_limits_and_guesses(method):
    """An iteration limit, a good initial guess and a zero load end the loop where they should."""
    spec = cantilever(20, 10, 10, method_options(method, 1e-10, (2, 1, 1)))
    spec.solver.fallback_max_iterations = -1
    p = EllipticProblem(spec)
    zd = p.to_dev(splitmix_uniform(p.num_nodes, 3, 0.2, 1.0))
    u, st = p.solution(zd)
    again, sa = p.solution(zd, u0=u)
    assert sa["iterations"] <= 1 and rel_l2(again.cpu().numpy(), u.cpu().numpy()) <= 1e-8
    opts = method_options(method, 1e-10, (2, 1, 1))
    opts.max_iterations, opts.fallback_max_iterations = 3, -1
    p.set_solver(opts)
    _, sl = p.solution(zd, raise_on_error=False)
    assert sl["rc"] == capi.NOT_CONVERGED and sl["iterations"] == 3
    still = cantilever(20, 10, 10, method_options(method, 1e-10, (2, 1, 1)))
    still.tractions = []
    q = EllipticProblem(still)
    u0, s0 = q.solution(zd)
    assert s0["iterations"] == 0 and not u0.any()
    bad = zd.clone()
    bad[17] = float("nan")
    p.set_solver(method_options(method, 1e-10, (2, 1, 1)))
    _, sn = p.solution(bad, raise_on_error=False)
    assert sn["rc"] == capi.NONFINITE


@pytest.mark.parametrize("size", [(2, 2, 2), (7, 3, 2), (24, 12, 12), (80, 40, 40), (90, 42, 43), (110, 53, 52)],
                         ids=lambda s: "x".join(map(str, s)))
def test_filter_cooperative_matches_launch_per_stage(size):
    """Scalar systems: one warp per slice, two slices per warp, and one size beyond the loop's range."""
    m = box_mesh(*size, 2.0, 1.0, 1.0)
    f = HelmholtzFilter(m.coords, m.connectivity, 0.08)
    c = f.to_dev(splitmix_uniform(m.num_nodes, 4))
    a, sa = f.solution(c)
    g, _ = f.criterion_gradient(c)
    f.set_timing(True)
    b, sb = f.solution(c)
    h, _ = f.criterion_gradient(c)
    assert abs(sa["iterations"] - sb["iterations"]) <= 2, (sa, sb)
    # both stop at 1e-12 and the filter's operator is well conditioned
    assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-10 and rel_l2(g.cpu().numpy(), h.cpu().numpy()) <= 1e-10


@pytest.mark.parametrize("size", [(4, 3, 3), (9, 5, 5), (13, 6, 6), (18, 9, 9), (21, 10, 10)], ids=lambda s: "x".join(map(str, s)))
def test_cluster_matches_launch_per_stage(size):
    """Systems that run as one thread-block cluster: 2, 8 and 16 CTAs, ragged shares, and the first size beyond;
    the scalar filter on the same meshes (and its own bars)."""
    spec = cantilever(*size, method_options("plain", 1e-10, (2, 1, 1)))
    z = splitmix_uniform(spec.coords.shape[0], 3, 0.2, 1.0)
    p = EllipticProblem(spec)
    f = HelmholtzFilter(spec.coords, spec.connectivity, 0.08)
    got = []
    for timing in (False, True):
        p.set_timing(timing)
        f.set_timing(timing)
        u, st = p.solution(p.to_dev(z))
        assert st["converged"] and st["fallback"] == 0 and st["relative_residual"] <= 1e-10, st
        got.append((st["iterations"], u.cpu().numpy(), f.solution(f.to_dev(z))[0].cpu().numpy()))
    (a, u, c), (b, v, d) = got
    assert abs(a - b) <= max(3, b // 20) and rel_l2(u, v) <= 1e-8 and rel_l2(c, d) <= 1e-10
    uo, _, _ = Oracle.from_spec(spec).solution_refined(z, tol=1e-13)
    assert rel_l2(u, uo) <= 1e-8


def test_multistep_sweep_beyond_the_cooperative_range():
    """The multi-step sweep kernel serves the systems that the cooperative loop leaves to it: the same
    arithmetic per row as one launch per step, so the same iterations and solution."""
    spec = cantilever(72, 34, 34, method_options("two-level-fp16", 1e-10, coarse_grid(72, 34, 34)))
    p = EllipticProblem(spec)
    zd = p.to_dev(splitmix_uniform(p.num_nodes, 3, 0.2, 1.0))
    got = []
    for steps in (0, 4, 7):
        spec.solver.sweep_steps = steps
        p.set_solver(spec.solver)
        u, st = p.solution(zd)
        assert st["converged"] and st["fallback"] == 0 and p.sweep_info()["steps_per_launch"] == max(1, steps)
        got.append((st["iterations"], u.cpu().numpy()))
    for it, u in got[1:]:
        assert it == got[0][0] and rel_l2(u, got[0][1]) <= 1e-14  # the bar of the small meshes' test


@pytest.mark.parametrize("size", [(112, 56, 56), (120, 60, 60)], ids=lambda s: "x".join(map(str, s)))
def test_sweep_on_both_sides_of_the_l2(size):
    """The FP16 sweep with a matrix that fits in the L2 and with one that is read evict-first: both solves meet
    the tolerance that the FP32 sweep's solve of the same system meets."""
    got = []
    for method in ("two-level-fp16", "two-level"):
        spec = cantilever(*size, method_options(method, 1e-10, coarse_grid(*size)))
        p = EllipticProblem(spec)
        u, st = p.solution(p.to_dev(splitmix_uniform(p.num_nodes, 3, 0.2, 1.0)))
        assert st["converged"] and st["fallback"] == 0 and st["relative_residual"] <= 1e-10, st
        got.append(u.cpu().numpy())
    assert rel_l2(*got) <= 1e-8


def _split(p, nb):
    out = np.zeros(6, np.int32)
    slices = (p.num_nodes + 31) // 32
    assert capi.lib.plato_test_pcg_split(slices, p.sell_info()["total_slots"], nb, 148, 1, out.ctypes.data_as(capi.i32p)) == capi.OK
    return {"per_cta": int(out[1]), "parts": int(out[2]), "in_smem": int(out[4])}


@pytest.mark.parametrize("size,per_cta,parts", [((13, 9, 9), 3, 5), ((20, 10, 10), 5, 3), ((40, 18, 16), 3, 5), ((48, 21, 20), 5, 3)],
                         ids=str)
def test_shares_that_leave_warps_over(size, per_cta, parts):
    """3 and 5 slices on the 16 warps of a CTA: 5 and 3 warps each and one left over, as a cluster and as a
    grid.  The bars of the other comparisons with the launch per stage."""
    spec = cantilever(*size, method_options("plain", 1e-10, (2, 1, 1)))
    z = splitmix_uniform(spec.coords.shape[0], 3, 0.2, 1.0)
    p = EllipticProblem(spec)
    assert _split(p, 3) == {"per_cta": per_cta, "parts": parts, "in_smem": 1}
    u, st = p.solution(p.to_dev(z))
    p.set_timing(True)
    v, sv = p.solution(p.to_dev(z))
    assert st["converged"] and sv["converged"] and abs(st["iterations"] - sv["iterations"]) <= max(3, sv["iterations"] // 20)
    assert rel_l2(u.cpu().numpy(), v.cpu().numpy()) <= 1e-8


def mirrored_box(nx, ny, nz):
    """A box whose hexes are cut like the mirror images of their neighbours: the cells of box_mesh's shape, but
    every other node has 26 neighbours, so that nearly every slice of 32 rows is 27 blocks wide."""
    m = box_mesh(nx, ny, nz, 2.0, 1.0, 1.0)
    n = np.array([nx + 1, ny + 1, nz + 1])
    at = np.stack(np.unravel_index(m.connectivity, n), -1)  # the cells of a hex are 6 in a row
    low = at.reshape(-1, 24, 3).min(1)[:, None, None, :]
    offset = (at.reshape(-1, 6, 4, 3) - low) ^ (low & 1)
    return m, np.ascontiguousarray(np.ravel_multi_index(tuple(np.moveaxis(low + offset, -1, 0)), n).reshape(-1, 4), np.int32)


def test_shares_that_leave_warps_over_from_l2():
    """5 slices a CTA with rows so wide that the matrix does not fit in shared memory."""
    m, conn = mirrored_box(48, 21, 20)
    fixed = np.nonzero(m.coords[:, 0] == 0.0)[0]
    dofs = (3 * fixed[:, None] + np.arange(3)).reshape(-1).astype(np.int32)
    on = m.coords[conn, 0] == 2.0
    cells = np.nonzero(on.sum(1) == 3)[0]
    local = np.nonzero(on[cells])[1].reshape(-1, 3)
    spec = ProblemSpec(m.coords, conn, 1.0, 0.3, 3.0, 1e-9, [(cells.astype(np.int32), local.astype(np.int32), (0.0, -1.0, 0.0))],
                       dofs, np.zeros(dofs.size), method_options("plain", 1e-10, (2, 1, 1)))
    z = splitmix_uniform(m.num_nodes, 3, 0.2, 1.0)
    p = EllipticProblem(spec)
    assert _split(p, 3) == {"per_cta": 5, "parts": 3, "in_smem": 0}
    u, st = p.solution(p.to_dev(z))
    p.set_timing(True)
    w, sw = p.solution(p.to_dev(z))
    assert st["converged"] and sw["converged"] and abs(st["iterations"] - sw["iterations"]) <= max(3, sw["iterations"] // 20)
    assert rel_l2(u.cpu().numpy(), w.cpu().numpy()) <= 1e-8


@pytest.mark.parametrize("size,per_cta", [((13, 9, 9), 3), ((18, 11, 10), 5), ((20, 11, 11), 6), ((24, 14, 11), 9),
                                          ((48, 21, 20), 5), ((50, 22, 20), 6), ((60, 26, 24), 9), ((62, 26, 25), 10)], ids=str)
def test_filter_shares_that_leave_warps_over(size, per_cta):
    """The scalar systems with 3 to 10 slices on the 32 warps of a CTA, as a cluster and as a grid."""
    m = box_mesh(*size, 2.0, 1.0, 1.0)
    f = HelmholtzFilter(m.coords, m.connectivity, 0.08)
    slices = (m.num_nodes + 31) // 32
    out = np.zeros(6, np.int32)
    assert capi.lib.plato_test_pcg_split(slices, 15 * 32 * slices, 1, 148, 1, out.ctypes.data_as(capi.i32p)) == capi.OK
    assert out[1] == per_cta and 32 % out[2] != 0
    c = f.to_dev(splitmix_uniform(m.num_nodes, 4))
    a, sa = f.solution(c)
    f.set_timing(True)
    b, sb = f.solution(c)
    assert abs(sa["iterations"] - sb["iterations"]) <= 2 and rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-10


# (method, size, CTA whose wait runs out, barrier, iterations of the launch).  Flexible CG of degree d: barriers 1 and 2
# are sums, d - 2 more (with a coarse space d - 1) belong to the sweep, 5 to the coarse solve, the last two are sums.
STALLS = [("plain", (30, 16, 16), 0, 1, 0), ("plain", (30, 16, 16), 3, 7, 0), ("plain", (40, 20, 20), 147, 40, 0),
          ("chebyshev", (20, 10, 10), 0, 3, 0), ("chebyshev", (20, 10, 10), 1, 10, 1), ("bf16", (26, 12, 12), 5, 18, 1),
          ("two-level", (20, 10, 10), 2, 14, 0), ("two-level-fp16", (40, 20, 20), 7, 22, 1), ("two-level-fp16", (40, 20, 20), 0, 22, 1)]


@pytest.mark.parametrize("method,size,cta,barrier,iterations", STALLS, ids=str)
def test_a_wait_that_runs_out(method, size, cta, barrier, iterations):
    """A wait that runs out, in the middle of an iteration or at the last barrier of a launch, ends the launch; the
    solve goes on with one launch per stage and meets its tolerance, and so do the handle's later solves."""
    spec = cantilever(*size, method_options(method, 1e-10, coarse_grid(*size)))
    z = splitmix_uniform(spec.coords.shape[0], 3, 0.2, 1.0)
    p = EllipticProblem(spec)
    zd = p.to_dev(z)
    v, _ = p.solution(zd)
    p.reset_instrumentation()
    _, sv = p.solution(zd)
    few = p.instrumentation()["launches"]
    assert capi.lib.plato_test_stall_next_grid(p.h, cta, barrier, iterations) == capi.OK
    for _ in range(2):
        p.reset_instrumentation()
        u, st = p.solution(zd)
        assert st["converged"] and st["fallback"] == 0 and st["relative_residual"] <= 1e-10, st
        assert p.instrumentation()["launches"] > few + st["iterations"]
        assert rel_l2(u.cpu().numpy(), v.cpu().numpy()) <= 1e-8
    assert st["iterations"] > 1 and sv["iterations"] > 1


def test_a_wait_that_runs_out_in_the_filter():
    m = box_mesh(48, 21, 20, 2.0, 1.0, 1.0)
    f = HelmholtzFilter(m.coords, m.connectivity, 0.08)
    c = f.to_dev(splitmix_uniform(m.num_nodes, 4))
    a, _ = f.solution(c)
    assert capi.lib.plato_test_stall_next_grid(f.h, 9, 6, 0) == capi.OK
    for _ in range(2):
        b, _ = f.solution(c)
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-10


@pytest.mark.parametrize("sms", [5, 4, 0])
@pytest.mark.parametrize("method", ["plain", "chebyshev", "two-level-fp16"])
def test_a_device_with_fewer_sms(method, sms):
    """80 slices on 5 SMs, the most that 16 warps each hold, on 4, which are too few, and on a device without
    cooperative launches: the same solution, by the launch per stage in the last two."""
    spec = cantilever(20, 10, 10, method_options(method, 1e-10, (2, 1, 1)))
    p = EllipticProblem(spec)
    zd = p.to_dev(splitmix_uniform(p.num_nodes, 3, 0.2, 1.0))
    p.solution(zd)
    p.reset_instrumentation()
    v, _ = p.solution(zd)
    few = p.instrumentation()["launches"]
    assert capi.lib.plato_test_grid_sms(p.h, sms) == capi.OK and capi.lib.plato_test_grid_sms(p.h, sms + 1) == capi.BAD_INPUT
    p.reset_instrumentation()
    u, st = p.solution(zd)
    assert st["converged"] and st["fallback"] == 0 and st["relative_residual"] <= 1e-10, st
    assert (p.instrumentation()["launches"] > few + st["iterations"]) == (sms < 5)
    assert rel_l2(u.cpu().numpy(), v.cpu().numpy()) <= 1e-8


@pytest.mark.parametrize("cells", [(20, 10, 10), (40, 20, 20)], ids=str)
def test_multistep_sweep_on_the_staged_loop(cells):
    """The multi-step sweep in every iteration of small systems, which leave it to the cooperative loop otherwise:
    launch lengths that do and do not divide the degree, a one-tile lag and a long one do the same arithmetic per row as one
    launch per step, so the same iterations and the same solution (the bar of the small meshes' other test)."""
    spec = cantilever(*cells, SolverOptions(tolerance=1e-10))
    p = EllipticProblem(spec)
    zd = p.to_dev(splitmix_uniform(p.num_nodes, 0x5EED0003))
    opts = SolverOptions(tolerance=1e-10, precision=capi.PRECISION_MIXED_FP16, chebyshev_degree=9, chebyshev_ratio=100.0,
                         coarse_cells=tuple(c // 10 for c in cells), sweep_steps=4)
    p.set_solver(opts)
    v, _ = p.solution(zd)
    assert p.sweep_info()["cooperative"]
    assert capi.lib.plato_test_grid_sms(p.h, 0) == capi.OK
    got = []
    for opts.sweep_steps, opts.sweep_lag in ((1, 0), (2, 0), (3, 0), (4, 0), (7, 1), (16, 0), (0, 0), (5, 300)):
        p.set_solver(opts)
        u, st = p.solution(zd)
        assert st["converged"] and st["fallback"] == 0, (opts, st)
        info = p.sweep_info()
        assert info["steps_per_launch"] == max(1, opts.sweep_steps) and not info["cooperative"]
        got.append((st["iterations"], u.cpu().numpy()))
    for it, u in got[1:]:
        assert it == got[0][0] and rel_l2(u, got[0][1]) <= 1e-14
    assert rel_l2(v.cpu().numpy(), got[0][1]) <= 1e-8


@pytest.mark.parametrize("size,mirrored,cooperative", [((72, 36, 35), False, 1), ((72, 36, 35), True, 0), ((90, 40, 38), True, 1)], ids=str)
def test_filter_of_wide_rows(size, mirrored, cooperative):
    """21 slices per SM run cooperatively with narrow rows and stay with the launch per stage with wide ones; 31 slices
    of wide rows per SM, two to a warp and read from L2, run cooperatively.  The bars of the other comparisons."""
    m, conn = mirrored_box(*size)
    f = HelmholtzFilter(m.coords, conn if mirrored else m.connectivity, 0.08)
    c = f.to_dev(splitmix_uniform(m.num_nodes, 4))
    a, sa = f.solution(c)
    used = np.zeros(1, np.int32)
    assert capi.lib.plato_get_loop_info(f.h, used.ctypes.data_as(capi.i32p)) == capi.OK and used[0] == cooperative
    f.set_timing(True)
    b, sb = f.solution(c)
    assert abs(sa["iterations"] - sb["iterations"]) <= 2 and rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-10
