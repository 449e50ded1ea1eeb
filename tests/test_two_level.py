"""The two-level factorization on K's fine rows (a KKT system in its natural
order) against the oracle, bit for bit, over the forms that its rule accepts
-- tile sizes, dense blocks, dropped entries, missing diagonals, long rows --
and next to them the forms that keep the general path: an unsymmetric
pattern, static pivots and a drop threshold on the same factor object."""
import numpy as np
import pytest

import culip_b200 as cb

torch = pytest.importorskip("torch")
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _kkt(n, m, A, rng, h=None, gamma=1e-6):
    """K = [[H, A'], [A, -gamma I]] as full symmetric CSR from a dense A (0 = no entry)."""
    h = rng.uniform(0.1, 10.0, n) if h is None else h
    K = np.zeros((n + m, n + m))
    K[np.arange(n), np.arange(n)] = h
    K[n:, :n] = A
    K[:n, n:] = A.T
    K[np.arange(n, n + m), np.arange(n, n + m)] = -gamma
    return _csr(K)


def _csr(K):
    rows, cols = np.nonzero(K)
    rp = np.zeros(len(K) + 1, np.int32)
    np.add.at(rp, rows + 1, 1)
    return np.cumsum(rp).astype(np.int32), cols.astype(np.int32), K[rows, cols]


def _random_a(n, m, density, rng):
    return np.where(rng.random((m, n)) < density, rng.standard_normal((m, n)), 0.0)


def _system(form):
    rng = np.random.default_rng(11)
    n, m, block = 150, 67, 8
    h = None
    if form.startswith("block"):
        block = int(form[5:])
        A = _random_a(n, m, 0.05, rng)
    elif form == "dense":  # every off-diagonal block dense
        A = _random_a(n, m, 1.0, rng)
    elif form == "mixed":  # some blocks dense, some sparse
        A = _random_a(n, m, 0.03, rng)
        A[8:24, 16:48] = rng.standard_normal((16, 32))
    elif form == "dropped":  # entries on both sides of the drop tolerance, some of whole rows
        A = _random_a(n, m, 0.06, rng) * 10.0 ** rng.uniform(-12, 0, (m, n))
        A[:, :16] *= 1e-14
        A[8:24, 40:56] = 1e-12 * rng.standard_normal((16, 16))  # dense blocks keep theirs
    elif form == "long":  # rows and columns well beyond a batch of loads
        A = _random_a(n, m, 0.02, rng)
        A[:, 3] = rng.standard_normal(m)
        A[5] = rng.standard_normal(n)
    elif form == "wide":  # a tile's run of U' beyond what is staged at once, over several chunks
        n, m, block = 900, 40, 32
        A = _random_a(n, m, 0.05, rng)
    elif form == "full32":  # full tiles of 32: more pairs than the two-level form takes
        n, m, block = 96, 64, 32
        A = _random_a(n, m, 1.0, rng)
    elif form == "tiny":  # pivots below the perturbation bound
        A = _random_a(n, m, 0.05, rng)
        h = rng.uniform(0.1, 10.0, n)
        h[::7] = 1e-9
    elif form == "swaps":  # wide-ranging H: many swaps and 2x2 candidates in the tiles
        A = _random_a(n, m, 0.12, rng)
        h = 10.0 ** rng.uniform(-5, 5, n) * np.where(rng.random(n) < 0.3, -1, 1)
        block = 32
    else:
        A = _random_a(n, m, 0.05, rng)
    rp, ci, v = _kkt(n, m, A, rng, h)
    if form == "nodiag":
        keep = np.ones(len(ci), bool)
        for i in range(0, n, 5):
            keep[rp[i]] = False
        rp, ci, v = _mask(rp, ci, v, keep)
    if form == "lower":  # the factor reads the upper triangle: other values below it change nothing
        rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
        v = np.where(ci < rows, 7.0, v)
    if form == "unsymmetric":  # nor do missing entries there
        rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
        rp, ci, v = _mask(rp, ci, v, (ci >= rows) | (rng.random(len(ci)) < 0.5))
    return rp, ci, v, cb.kkt_blocking(n, m, block)


def _mask(rp, ci, v, keep):
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))[keep]
    out = np.zeros(len(rp), np.int32)
    np.add.at(out, rows + 1, 1)
    return np.cumsum(out).astype(np.int32), ci[keep], v[keep]


def _same_factor(F, OF):
    ge, oe = F.export(), OF.export()
    for k in ("blk_nnz", "blk_off", "idx", "val", "tri", "is_piv", "perm", "got_extra"):
        assert np.array_equal(oe[k], ge[k]), k


def _same_applies(F, OF, n, dtype):
    b = np.random.default_rng(3).standard_normal(n).astype(dtype)
    for stage in (cb.LEFT, cb.MIDDLE, cb.RIGHT):
        got = F.apply(stage, torch.from_numpy(b).cuda()).cpu().numpy()
        assert np.array_equal(got, OF.apply(stage, b)), stage


FORMS = ["block1", "block2", "block7", "block31", "block32", "dense", "mixed", "dropped", "long", "tiny", "swaps",
         "wide", "full32", "nodiag", "lower", "unsymmetric"]


@pytest.mark.parametrize("prec", [cb.F64, cb.F32])
@pytest.mark.parametrize("form", FORMS)
def test_two_level_factor_exact(form, prec):
    dtype = np.float64 if prec == cb.F64 else np.float32
    rp, ci, v, bs = _system(form)
    n = len(rp) - 1
    S = oracle.Sym(rp, ci, bs, 0, 1.0, dtype)
    F = cb.Factor(cb.Pattern(cb.Handle(0), rp, ci, bs, 0, 1.0, prec))
    vals = torch.from_numpy(v.astype(dtype)).cuda()
    for pivot in (cb.PIV_BK, cb.PIV_ROOK):
        F.compute(vals, pivot=pivot)
        OF = S.factor(v.astype(dtype), pivot=pivot)
        _same_factor(F, OF)
        _same_applies(F, OF, n, dtype)


def test_routes_alternate_on_one_factor():
    """Bunch-Kaufman, static pivots, a threshold and Jacobi sweeps in turn on
    one factor object: each as the oracle's, whatever ran before."""
    rp, ci, v, bs = _system("block7")
    n = len(rp) - 1
    S = oracle.Sym(rp, ci, bs, 0, 1.0)
    F = cb.Factor(cb.Pattern(cb.Handle(0), rp, ci, bs, 0, 1.0, cb.F64))
    vals = torch.from_numpy(v).cuda()
    ones = np.ones(n, np.int32)
    for pivot, threshold in ((cb.PIV_BK, 0.0), (cb.PIV_STATIC, 0.0), (cb.PIV_BK, 1e-2), (cb.PIV_ROOK, 0.0)):
        F.compute(vals, ones if pivot == cb.PIV_STATIC else None, pivot, threshold)
        OF = S.factor(v, ones if pivot == cb.PIV_STATIC else None, pivot, threshold)
        _same_factor(F, OF)
        _same_applies(F, OF, n, np.float64)
        assert F.info()["u_nnz"] == sum(int(r != c) * k for r, c, k in _block_counts(F, S))
    F.set_solve_algorithm(cb.SOLVE_JACOBI, 2)
    b = np.random.default_rng(4).standard_normal(n)
    for stage in (cb.LEFT, cb.RIGHT):
        got = F.apply(stage, torch.from_numpy(b).cuda()).cpu().numpy()
        assert np.array_equal(got, OF.apply(stage, b, 2))


def _block_counts(F, S):
    """(block row, block column, stored non-zeros) of every block of the last factor."""
    e, p = F.export(), F.pattern.export()
    rows = np.repeat(np.arange(len(p["coarse_off"]) - 1), np.diff(p["coarse_off"]))
    for b in range(len(rows)):
        vals = e["val"][e["blk_off"][b]: e["blk_off"][b + 1]]
        yield rows[b], p["coarse_col"][b], int(np.count_nonzero(vals))
