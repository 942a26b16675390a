"""The solve and the V-cycle's bottom in one thread-block cluster (the default for hierarchies that
fit): the passes of a cluster follow the launched ones step by step, so the V-cycle equals theirs and
the FP64 oracle's bit for bit (kernel/solver/multigrid.hpp:1713-2000); a solve differs from theirs
only in the order of the sums r.z, p.Ap and ||r|| (kernel/solver/pcg.hpp:159-286)."""
import numpy as np
import pytest

from helpers import rel_err, to_oracle_levels

pytestmark = pytest.mark.gpu


# one block (level 4) and sixteen; the largest levels that fit as a whole (2D FP64: 7) and the first
# that do not (8: the bottom below a launched top level); a numbering without bands; odd step counts
@pytest.mark.parametrize("level,dim,ordering,precision,steps", [
    (3, 2, "native", "f64", 2), (4, 2, "native", "f64", 1), (5, 2, "rcm", "f32", 3), (6, 2, "native", "f32_bf16", 2),
    (7, 2, "native", "f64", 2), (7, 2, "rcm", "f64", 2), (8, 2, "native", "f64", 2), (8, 2, "rcm", "f32", 2),
    (3, 3, "native", "f64", 2), (4, 3, "rcm", "f32_bf16", 3), (5, 3, "native", "f32", 2)])
def test_cluster_equals_launched_passes(featlib, cuda, oracle_lib, level, dim, ordering, precision, steps):
    import torch
    from featb200 import assembly as AS
    fb = featlib
    levels, b = AS.poisson_hierarchy(level, dim, rhs="gauss", gauss=AS.gauss_params(level, dim))
    kw = dict(precision=precision, ordering=ordering, steps=steps)
    s = fb.build_pcg_multigrid(levels, **kw)
    ref = fb.build_pcg_multigrid(levels, tail_rows=301, **kw)       # chooses its passes: no cluster plan
    rng = np.random.default_rng(level)
    x0 = rng.standard_normal(b.size) * (b != 0)
    # FP64: sums in another order, 1e-12 of the solution; lower precisions: the scale of the defect is a
    # power of two, so the sums differ the same way, and the solves stop at 1e-8 of the first defect
    tol = 1e-12 if precision == "f64" else 1e-9
    for scale in (1.0, 3.0):
        if scale != 1.0:
            for l, L in enumerate(levels):
                v = torch.tensor(L["matrix"].val * scale, device="cuda")
                s.update_matrix(l, v)
                ref.update_matrix(l, v)
        z = s.apply_precond(fb.DenseVector(b)).elements
        assert np.array_equal(z, ref.apply_precond(fb.DenseVector(b)).elements)
        if precision == "f64" and steps == 2 and scale == 1.0:
            assert np.array_equal(z, oracle_lib.MultigridPCG(to_oracle_levels(levels), 0.7, 2).vcycle(b))
        xs = []
        for t in (s, ref):
            x = torch.tensor(x0, device="cuda")                   # a non-zero initial guess
            assert t.correct_device(x, torch.tensor(b, device="cuda")) == fb.Status.success
            xs.append(x.cpu().numpy())
        assert s.get_num_iter() == ref.get_num_iter()
        assert s.get_def_initial() == pytest.approx(ref.get_def_initial(), rel=1e-13)
        assert rel_err(xs[0], xs[1]) <= tol
    one = [fb.build_pcg_multigrid(levels, max_iter=1, **kw), fb.build_pcg_multigrid(levels, max_iter=1, tail_rows=301, **kw)]
    xs = []
    for t in one:
        x = torch.tensor(b, device="cuda")
        assert t.correct_device(x, x) == fb.Status.max_iter       # solution and right-hand side in one array
        assert t.get_num_iter() == 1
        xs.append(x.cpu().numpy())
    assert rel_err(xs[0], xs[1]) <= tol
    zero = torch.zeros(b.size, dtype=torch.float64, device="cuda")
    assert s.correct_device(zero, zero.clone()) == fb.Status.success and s.get_num_iter() == 0
    bad = torch.full((b.size,), float("nan"), dtype=torch.float64, device="cuda")
    assert s.correct_device(torch.zeros_like(bad), bad) == fb.Status.aborted


@pytest.mark.parametrize("precision", ["f64", "f32_bf16"])
def test_update_follows_in_one_launch_per_array(featlib, cuda, precision):
    """fb_solver_update_matrix launches what a solver without a cluster plan launches (values, in FP32 modes the
    FP64 copy, diagonal): the plan's image is rewritten in the last of them."""
    import torch
    from featb200 import assembly as AS
    fb = featlib
    levels, _ = AS.poisson_hierarchy(6, 2, rhs="sine")
    count = []
    for kw in ({}, {"tail_rows": 301}):
        s = fb.build_pcg_multigrid(levels, precision=precision, **kw)
        c0 = fb.launch_count()
        for l, L in enumerate(levels):
            s.update_matrix(l, torch.tensor(L["matrix"].val, device="cuda"))
        count.append(fb.launch_count() - c0)
    assert count[0] == count[1]


@pytest.mark.parametrize("precision", ["f64", "f32_bf16"])
def test_more_diagonals_than_entries_per_row(featlib, cuda, precision):
    """Diagonal storage with diagonals that few rows have: the cluster's rows hold their own entries only, as
    long as the longest of them; solves agree with the launched passes' before and after an update."""
    import scipy.sparse as sp
    import torch
    from featb200 import assembly as AS
    fb = featlib
    levels, b = AS.poisson_hierarchy(5, 2, rhs="gauss", gauss=AS.gauss_params(5, 2))
    for L in levels[:-2]:
        A, n = L["matrix"].to_scipy().tocsr(), 2 ** L["level"] + 1
        i = np.array([r * n + 1 + 2 * (r % 2) for r in range(1, n - 1)])   # couples (1 or 3, r) with 3 further on
        E = sp.coo_matrix((np.full(i.size, -0.1), (i, i + 3)), shape=A.shape)
        W = (A + E + E.T + sp.diags(np.asarray((-E - E.T).sum(axis=1)).ravel())).tocsr()
        W.sort_indices()
        L["matrix"] = fb.SparseMatrixCSR.from_scipy(W)
        p = fb.storage_plan(L["matrix"], L["filter"].indices)
        assert p["kind"] == "diagonal" and p["diagonals"] == 11 and np.diff(W.indptr).max() == 10
    s, ref = (fb.build_pcg_multigrid(levels, precision=precision, **kw) for kw in ({}, {"tail_rows": 301}))
    for scale in (1.0, 3.0):
        if scale != 1.0:
            for l, L in enumerate(levels):
                v = torch.tensor(L["matrix"].val * scale, device="cuda")
                s.update_matrix(l, v)
                ref.update_matrix(l, v)
        xs = []
        for t in (s, ref):
            x = torch.zeros(b.size, dtype=torch.float64, device="cuda")
            assert t.correct_device(x, torch.tensor(b, device="cuda")) == fb.Status.success
            xs.append(x.cpu().numpy())
        assert s.get_num_iter() == ref.get_num_iter()
        assert rel_err(xs[0], xs[1]) <= (1e-12 if precision == "f64" else 1e-9)


def test_cluster_switch(featlib, cuda):
    """cluster_rows below 0 keeps clusters out with every other option at its default: the launched passes and the
    tail kernel, bit for bit those of a configuration that chooses its passes."""
    import torch
    from featb200 import assembly as AS
    fb = featlib
    levels, b = AS.poisson_hierarchy(5, 2, rhs="gauss", gauss=AS.gauss_params(5, 2))
    xs, launches = [], []
    for kw in ({}, {"cluster_rows": -1}, {"tail_rows": 301}):
        s = fb.build_pcg_multigrid(levels, **kw)
        x = torch.zeros(b.size, dtype=torch.float64, device="cuda")
        c0 = fb.launch_count()
        assert s.correct_device(x, torch.tensor(b, device="cuda")) == fb.Status.success
        launches.append(fb.launch_count() - c0)
        xs.append(x.cpu().numpy())
    assert launches[0] == 1 and launches[1] == launches[2] > 1
    assert np.array_equal(xs[1], xs[2]) and rel_err(xs[0], xs[1]) <= 1e-12


@pytest.mark.parametrize("kw", [{}, {"cluster_rows": -1}])
def test_min_iter_above_max_iter(featlib, cuda, kw):
    """min_iter is tested before max_iter: a solve takes min_iter iterations."""
    import torch
    from featb200 import _lib, assembly as AS
    fb = featlib
    levels, b = AS.poisson_hierarchy(5, 2, rhs="gauss", gauss=AS.gauss_params(5, 2))
    s = fb.build_pcg_multigrid(levels, max_iter=2, **kw)
    _lib.check(_lib.lib().fb_solver_set_iteration_limits(s._s, 9, 2))
    x = torch.zeros(b.size, dtype=torch.float64, device="cuda")
    assert s.correct_device(x, torch.tensor(b, device="cuda")) == fb.Status.success
    assert s.get_num_iter() == 9
