"""Batches on the whole grid whose large systems stop first: the small ones that
are left are finished by a CTA each, from the iteration they had reached.  A
system's result is the one that it has alone, bit for bit, wherever the others
stop -- after some iterations, at the first test, or at once."""
import numpy as np
import pytest

import culip_b200 as cb

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _system(n, spread, seed, block=16):
    rp, ci, v = cb.kkt_generate(n, n // 2, 5, 16, 1 / spread, spread, delta=1e-6, gamma=1e-6, seed=seed)
    return rp, ci, v, cb.kkt_blocking(n, n // 2, block)


def _solve(systems, rhs, precision, tol, max_it, graph=False):
    rp, ci, v, bs, off = cb.union_systems(systems)
    h = cb.Handle(0)
    P = cb.Pattern(h, rp, ci, bs, 0, 1.0, precision, system_row_offsets=off)
    F, B = cb.Factor(P), cb.Batch(P, off)
    d = [torch.from_numpy(a).cuda() for a in (rp, ci, v)]
    vals = d[2] if precision == cb.F64 else d[2].float()
    A = cb.CsrOperator(h, *d)
    b = torch.from_numpy(np.concatenate(rhs)).cuda()
    x = torch.full_like(b, 7.0)
    if graph:
        for _ in range(3):  # ordinary, then two replays
            x.fill_(7.0)
            res, its, st = cb.batch_factor_solve_graph(B, A, F, vals, b, x, tol, max_it)
    else:
        F.compute(vals)
        res, its, st = cb.batch_sqmr_solve(B, A, F, b, x, tol, max_it)
    x = x.cpu().numpy()
    return [(x[off[k]:off[k + 1]], res[k], its[k], st[k]) for k in range(len(systems))]


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("precision", [cb.F64, cb.F32])
@pytest.mark.parametrize("large", ["easy", "zero rhs", "nan rhs"])
def test_small_systems_outlast_the_large_one(large, precision, graph):
    # rows of 390, 1350, 3000 and 60, and 12 000 in their midst
    systems = [_system(n, 1e5, 3 + k) for k, n in enumerate((260, 900, 2000, 40))]
    systems.insert(2, _system(8000, 4.0, 9))
    rhs = [cb.normal_vector(11 + k, len(s[0]) - 1) for k, s in enumerate(systems)]
    if large == "zero rhs":
        rhs[2] = np.zeros_like(rhs[2])
    elif large == "nan rhs":
        rhs[2][5] = np.nan
    tol, max_it = 1e-7, 300
    together = _solve(systems, rhs, precision, tol, max_it, graph)
    if large == "easy":  # what the test is about
        assert together[2][2] < min(together[k][2] for k in (0, 1, 3))
    for k, (s, b) in enumerate(zip(systems, rhs)):
        x, res, its, st = _solve([s], [b], precision, tol, max_it)[0]
        assert (its, st) == together[k][2:], k
        assert np.array_equal(res, together[k][1], equal_nan=True), k
        assert np.array_equal(x, together[k][0], equal_nan=True), k
