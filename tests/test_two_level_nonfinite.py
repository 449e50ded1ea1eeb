"""Values that are not finite in the factorization on K's fine rows, and its
stages in place.

The same upper triangle without one entry below the diagonal is a pattern that
keeps the general path, which multiplies whole blocks: a NaN or an infinity
meets their zeros there, so that a factor of such a K is not finite in whole
rows of a tile.  The fine rows have to give the same factor and the same stages,
NaN for NaN."""
import numpy as np
import pytest

import culip_b200 as cb
from test_two_level import _mask, _system

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

STAGES = (cb.LEFT, cb.MIDDLE, cb.RIGHT)
KINDS = ["finite", "nan diagonal", "inf diagonal", "nan entry", "inf entry", "nan tile", "inf tile", "huge", "tiny",
         "half nan"]


def _pair(form, precision):
    """(factor on fine rows, factor on the general path, which values the second takes, system)"""
    rp, ci, v, bs = _system(form)
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    keep = np.ones(len(ci), bool)
    keep[np.flatnonzero(ci < rows)[0]] = False
    fewer_rp, fewer_ci, _ = _mask(rp, ci, v, keep)
    h = cb.Handle(0)
    F = cb.Factor(cb.Pattern(h, rp, ci, bs, 0, 1.0, precision))
    G = cb.Factor(cb.Pattern(h, fewer_rp, fewer_ci, bs, 0, 1.0, precision))
    launches = []
    for M, values in ((F, v), (G, v[keep])):
        h.launch_count(reset=True)
        M.compute(values)
        launches.append(h.launch_count())
    assert launches[0] == 3 and launches[1] > 3  # each on its path
    return F, G, keep, (rp, ci, v, rows)


def _values(kind, system, n0, dtype):
    rp, ci, v, rows = system
    w = v.astype(dtype).copy()
    rng = np.random.default_rng(3)
    diagonal = np.flatnonzero((ci == rows) & (rows < n0))
    entries = np.flatnonzero((rows < n0) & (ci >= n0))
    tile = np.flatnonzero((rows >= n0) & (ci >= rows))
    value = np.nan if kind.startswith("nan") else np.inf
    if kind.endswith("diagonal"):
        w[rng.choice(diagonal, 2, replace=False)] = value
    elif kind.endswith("entry"):
        w[rng.choice(entries, 3, replace=False)] = value
    elif kind.endswith("tile"):
        w[rng.choice(tile, 2, replace=False)] = value
    elif kind == "huge":  # finite, with products that are not
        w[rng.choice(entries, 9, replace=False)] = np.finfo(dtype).max / 10
    elif kind == "tiny":  # below the pivots' bound, and denormal entries
        w[rng.choice(diagonal, 5, replace=False)] = 1e-9
        w[rng.choice(entries, 20, replace=False)] = np.finfo(dtype).tiny / 4
    elif kind == "half nan":
        w[rng.choice(entries, len(entries) // 2, replace=False)] = np.nan
    return w


def _rows_of_level_0(form):
    return {"wide": 900}.get(form, 150)


@pytest.mark.parametrize("precision", [cb.F64, cb.F32])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("form", ["block1", "block7", "block32", "swaps", "nodiag", "tiny"])
def test_not_finite_as_the_general_path(form, kind, precision):
    dtype = np.float64 if precision == cb.F64 else np.float32
    F, G, keep, system = _pair(form, precision)
    w = _values(kind, system, _rows_of_level_0(form), dtype)
    n = len(system[0]) - 1
    b = torch.from_numpy(np.random.default_rng(1).standard_normal(n).astype(dtype)).cuda()
    for values in (w, system[2].astype(dtype)):  # and a finite K after it on the same factor
        for pivot in (cb.PIV_BK, cb.PIV_ROOK):
            F.compute(torch.from_numpy(values).cuda(), pivot=pivot)
            G.compute(torch.from_numpy(values[keep]).cuda(), pivot=pivot)
            got, want = F.export(), G.export()
            assert sorted(got["perm"]) == list(range(n))
            for k in ("blk_nnz", "blk_off", "idx", "is_piv", "perm"):
                assert np.array_equal(got[k], want[k]), k
            for k in ("val", "tri"):
                assert np.array_equal(got[k], want[k], equal_nan=True), k
            for stage in STAGES:
                x, y = F.apply(stage, b), G.apply(stage, b)
                assert np.array_equal(x.cpu().numpy(), y.cpu().numpy(), equal_nan=True), stage


@pytest.mark.parametrize("kind", ["nan diagonal", "inf diagonal", "nan entry", "inf entry", "half nan"])
@pytest.mark.parametrize("form", ["mixed", "wide"])
def test_dense_blocks_stay_not_finite(form, kind):
    """Dense blocks also fill in zeros of K that the fine rows have no place
    for: D^-1 and the whole solve with M are not finite all the same."""
    F, G, keep, system = _pair(form, cb.F64)
    w = _values(kind, system, _rows_of_level_0(form), np.float64)
    b = torch.from_numpy(np.random.default_rng(1).standard_normal(len(system[0]) - 1)).cuda()
    F.compute(torch.from_numpy(w).cuda())
    G.compute(torch.from_numpy(w[keep]).cuda())
    finite = []
    for M in (F, G):
        x = b
        for stage in STAGES:
            x = M.apply(stage, x)
        finite.append(bool(torch.isfinite(x).all()))
    assert finite[0] == finite[1]


@pytest.mark.parametrize("precision", [cb.F64, cb.F32])
@pytest.mark.parametrize("form", ["block1", "block7", "block32", "swaps", "long", "wide", "mixed"])
def test_stages_in_place(form, precision):
    dtype = np.float64 if precision == cb.F64 else np.float32
    rp, ci, v, bs = _system(form)
    F = cb.Factor(cb.Pattern(cb.Handle(0), rp, ci, bs, 0, 1.0, precision))
    F.compute(torch.from_numpy(v.astype(dtype)).cuda())
    b = np.random.default_rng(2).standard_normal(len(rp) - 1).astype(dtype)
    for stage in STAGES:
        want = F.apply(stage, torch.from_numpy(b).cuda())
        x = torch.from_numpy(b).cuda()
        F.apply(stage, x, x)
        assert torch.equal(x, want), stage
