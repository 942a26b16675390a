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
