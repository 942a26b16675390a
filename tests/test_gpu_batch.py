"""Batched uneven instances (fb_batch_*): every instance must follow its own single-system solve
(same iterations, FP64 results within 1e-12), including the reference's own problems, and the FP32
form stays within 1e-7 of FP64 at residual 1e-8."""
import numpy as np
import pytest

from helpers import load_golden, rel_err, to_lafem_levels

pytestmark = pytest.mark.gpu


def _family(levels_list, seed0=300, kappa=True):
    """Config-4 style instances: kappa = exp(random field), 8-Gaussian right-hand side."""
    from featb200 import assembly as AS
    out = []
    for k, L in enumerate(levels_list):
        field = AS.field_params(seed0 + 2 * k) if kappa else None
        lv, b = AS.poisson_hierarchy(L, 2, rhs="gauss", gauss=AS.gauss_params(seed0 + 2 * k + 1, 2), field=field)
        out.append((lv, b))
    return out


@pytest.mark.parametrize("ordering", ["native", "rcm"])
def test_batch_fp64_matches_single(featlib, cuda, ordering):
    fb = featlib
    inst = _family([4, 6, 3, 5, 4, 2])
    hs = [fb.build_hierarchy(lv) for lv, _ in inst]
    bat = fb.BatchPCG(hs, ordering=ordering)
    rhs = np.concatenate([b for _, b in inst])
    X = bat.split(bat.solve(np.zeros_like(rhs), rhs))
    for k, (lv, b) in enumerate(inst):
        s = fb.build_pcg_multigrid(lv, ordering=ordering)
        x = fb.DenseVector(b.size)
        assert fb.solve(s, x, fb.DenseVector(b)) == fb.Status.success
        assert bat.statuses()[k] == fb.Status.success
        assert bat.iterations()[k] == s.get_num_iter()
        assert rel_err(X[k], x.elements) <= 1e-12


def test_batch_reproduces_reference(featlib, cuda):
    """Instances straight from the reference's fixtures (reference numbering, noisy transfer
    matrices): each matches the reference's own solution."""
    fb = featlib
    names = ["c1_L4", "c1_L5", "gauss2d_L5", "kappa2d_L4"]
    gs = [load_golden(n) for n in names]
    hs = [fb.build_hierarchy(to_lafem_levels(g["levels"])) for g in gs]
    bat = fb.BatchPCG(hs)
    rhs = np.concatenate([g["rhs"] for g in gs])
    X = bat.split(bat.solve(np.zeros_like(rhs), rhs))
    for k, g in enumerate(gs):
        assert bat.iterations()[k] == g["summary"]["iters"]
        assert rel_err(X[k], g["sol"]) <= 1e-12


def test_batch_fp32_error(featlib, cuda):
    fb = featlib
    inst = _family([5, 7, 6, 8, 5, 9, 7, 6])
    hs = [fb.build_hierarchy(lv) for lv, _ in inst]
    rhs = np.concatenate([b for _, b in inst])
    b64 = fb.BatchPCG(hs, precision="f64")
    X64 = b64.split(b64.solve(np.zeros_like(rhs), rhs))
    b32 = fb.BatchPCG(hs, precision="f32")
    X32 = b32.split(b32.solve(np.zeros_like(rhs), rhs))
    for k, (lv, b) in enumerate(inst):
        assert b32.statuses()[k] == fb.Status.success
        A = lv[0]["matrix"].to_scipy()
        r = b - A @ X32[k]
        r[lv[0]["filter"].indices.astype(np.int64)] = 0.0
        assert np.linalg.norm(r) <= 1.05e-8 * np.linalg.norm(b)
        assert rel_err(X32[k], X64[k]) <= 1e-7


def test_batch_converged_instances_stop(featlib, cuda):
    """An instance with a zero right-hand side stops at iteration 0 while the others continue."""
    fb = featlib
    inst = _family([4, 5], kappa=False)
    hs = [fb.build_hierarchy(lv) for lv, _ in inst]
    bat = fb.BatchPCG(hs)
    rhs = np.concatenate([np.zeros_like(inst[0][1]), inst[1][1]])
    X = bat.split(bat.solve(np.zeros_like(rhs), rhs))
    assert bat.iterations()[0] == 0 and np.all(X[0] == 0)
    assert bat.statuses()[1] == fb.Status.success and bat.iterations()[1] > 0


@pytest.mark.parametrize("rows_per_block", [0, 64, 512])
def test_batch_rows_per_block(featlib, cuda, rows_per_block):
    """The autotuner (0) picks a block size per level from 64..512; any choice gives the same
    iterations and solutions as the single-system solves (block sizes change only which threads
    run which rows)."""
    fb = featlib
    inst = _family([5, 7, 3, 6], seed0=500)
    hs = [fb.build_hierarchy(lv) for lv, _ in inst]
    bat = fb.BatchPCG(hs, rows_per_block=rows_per_block)
    rpb = bat.rows_per_block()
    assert len(rpb) == 7
    if rows_per_block:
        assert np.all(rpb == rows_per_block)
    else:
        assert set(rpb.tolist()) <= {64, 128, 256, 512}
    rhs = np.concatenate([b for _, b in inst])
    X = bat.split(bat.solve(np.zeros_like(rhs), rhs))
    for k, (lv, b) in enumerate(inst):
        s = fb.build_pcg_multigrid(lv)
        x = fb.DenseVector(b.size)
        assert fb.solve(s, x, fb.DenseVector(b)) == fb.Status.success
        assert bat.iterations()[k] == s.get_num_iter()
        assert rel_err(X[k], x.elements) <= 1e-12


def test_batch_tunes_launched_levels_only(featlib, cuda):
    """Levels 1 to 3 of these instances run in the bottom kernel, with level 4 on top of it: 28 timed launches each
    for levels 4, 5 and 6 (after one that opens the instances)."""
    fb = featlib
    hs = [fb.build_hierarchy(lv) for lv, _ in _family([5, 6])]
    count = []
    for rows_per_block in (0, 64):
        c0 = fb.launch_count()
        fb.BatchPCG(hs, rows_per_block=rows_per_block)
        count.append(fb.launch_count() - c0)
    assert count[0] - count[1] == 1 + 3 * 28


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_batch_many_instances_per_block(featlib, cuda, precision):
    """Enough small instances (300 of levels 3 to 5) that a block's range of rows holds several of
    them: the per-instance sums are handed over between warps of one instance and the next.  Equal
    instances (every third) must take the same iterations, and FP64 solutions match single solves."""
    fb = featlib
    inst = _family([5, 3, 4])
    hs = [fb.build_hierarchy(lv) for lv, _ in inst]
    bat = fb.BatchPCG(hs * 100, precision=precision)
    rhs = np.concatenate([b for _, b in inst] * 100)
    X = bat.split(bat.solve(np.zeros_like(rhs), rhs))
    assert all(st == fb.Status.success for st in bat.statuses())
    for k, (lv, b) in enumerate(inst):
        s = fb.build_pcg_multigrid(lv)
        x = fb.DenseVector(b.size)
        assert fb.solve(s, x, fb.DenseVector(b)) == fb.Status.success
        assert len(set(bat.iterations()[k::3])) == 1
        for j in (k, 150 + k, 297 + k):
            assert rel_err(X[j], x.elements) <= (1e-12 if precision == "f64" else 1e-7)


# the bottom kernel's range: no level of its own (a top on level 2), one, four (289 rows) and the most
# with a level of 1,089 rows left to launched passes; one instance and more than one block per SM holds;
# three smoothing steps (the correction's buffers change places)
@pytest.mark.parametrize("levels,ordering,precision,steps", [
    ([2, 3], "native", "f64", 2), ([3], "rcm", "f64", 3), ([5, 6, 5], "native", "f64", 2), ([6, 7], "rcm", "f32_bf16", 2),
    ([5, 6], "native", "f32", 3), ([5] * 200 + [6], "native", "f32", 2)])
def test_batch_bottom_kernel(featlib, cuda, levels, ordering, precision, steps):
    """Instances agree with their single solves at every depth of the levels below the lowest top."""
    fb = featlib
    inst = _family(sorted(set(levels)))
    by = dict(zip(sorted(set(levels)), inst))
    single = {}
    for L, (lv, b) in by.items():
        s = fb.build_pcg_multigrid(lv, ordering=ordering, precision=precision, steps=steps)
        x = fb.DenseVector(b.size)
        assert fb.solve(s, x, fb.DenseVector(b)) == fb.Status.success
        single[L] = (x.elements.copy(), s.get_num_iter())
    hs = {L: fb.build_hierarchy(lv, steps=steps) for L, (lv, _) in by.items()}
    bat = fb.BatchPCG([hs[L] for L in levels], ordering=ordering, precision=precision)
    rhs = np.concatenate([by[L][1] for L in levels])
    X = bat.split(bat.solve(np.zeros_like(rhs), rhs))
    for k, L in enumerate(levels):
        assert bat.statuses()[k] == fb.Status.success
        assert bat.iterations()[k] == single[L][1]
        # the order of the PCG's sums differs
        assert rel_err(X[k], single[L][0]) <= (1e-12 if precision == "f64" else 1e-9)

def _coarse_first(levels, dim=2):
    """The hierarchy with every mesh's vertices numbered coarse vertices first: no level is lexicographic, and
    from 2D level 8 on column offsets leave the 16-bit range."""
    import featb200 as fb

    def order(level):
        idx = np.indices((2 ** level + 1,) * dim).reshape(dim, -1)
        age = np.zeros(idx.shape[1], dtype=np.int64)
        for lv in range(level):
            age += np.any(idx % (1 << (level - lv)) != 0, axis=0)
        return np.argsort(age, kind="stable")

    def permuted(m, rows, cols):
        return fb.SparseMatrixCSR.from_scipy(m.to_scipy()[rows][:, cols])

    out = []
    for d in levels:
        o = order(d["level"])
        place = np.argsort(o).astype(np.uint64)
        e = {"matrix": permuted(d["matrix"], o, o), "level": d["level"],
             "filter": fb.UnitFilter(np.sort(place[d["filter"].indices.astype(np.int64)]))}
        if "transfer" in d:
            c = order(d["level"] - 1)
            e["transfer"] = fb.Transfer(permuted(d["transfer"].get_mat_prol(), o, c),
                                        permuted(d["transfer"].get_mat_rest(), c, o))
        out.append(e)
    return out, order(levels[0]["level"])


def _widened(levels, c=0.05):
    """A + c A A on every level (boundary rows and columns of the product zero): 25 entries per interior row."""
    import scipy.sparse as sp
    import featb200 as fb
    out = []
    for d in levels:
        A = d["matrix"].to_scipy().tocsr()
        inner = np.ones(A.shape[0])
        inner[d["filter"].indices.astype(np.int64)] = 0.0
        A0 = sp.diags(inner) @ A @ sp.diags(inner)
        W = (A + c * (A0 @ A0)).tocsr()
        W.sort_indices()
        out.append(dict(d, matrix=fb.SparseMatrixCSR.from_scipy(W)))
    return out


# top matrices whose staged start needs more than 48 KB of shared memory: nine entries with 32-bit columns
# (55,296 bytes), and rows of up to 25 entries with 16-bit ones
@pytest.mark.parametrize("level,wide", [(8, False), (6, True)])
@pytest.mark.parametrize("use_graph", [True, False])
def test_batch_large_staged_start(featlib, cuda, level, wide, use_graph):
    """Instances numbered coarse vertices first match their single solves."""
    from featb200 import assembly as AS
    fb = featlib
    lex, b = AS.poisson_hierarchy(level, 2, rhs="gauss", gauss=AS.gauss_params(level, 2))
    levels, o = _coarse_first(_widened(lex) if wide else lex)
    b = b[o]
    plan = fb.storage_plan(levels[0]["matrix"], levels[0]["filter"].indices)
    assert plan["kind"] != "diagonal" and plan["narrow"] == wide and plan["width"] == (25 if wide else 9), plan
    s = fb.build_pcg_multigrid(levels)
    x = fb.DenseVector(b.size)
    assert fb.solve(s, x, fb.DenseVector(b)) == fb.Status.success
    h = fb.build_hierarchy(levels)
    bat = fb.BatchPCG([h, h], use_graph=use_graph)
    X = bat.split(bat.solve(np.zeros(2 * b.size), np.concatenate([b, b])))
    for k in range(2):
        assert bat.statuses()[k] == fb.Status.success
        assert bat.iterations()[k] == s.get_num_iter()
        assert rel_err(X[k], x.elements) <= 1e-12
