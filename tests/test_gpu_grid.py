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
from platoanalyze_b200.problem import EllipticProblem, HelmholtzFilter, SolverOptions
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
