"""The right stage of a two-level factor over rows of U on both sides of a batch
of loads, for either batch: rows that are long on average take 16 entries at a
time, others 8.  Both against the oracle, bit for bit."""
import numpy as np
import pytest

import culip_b200 as cb

torch = pytest.importorskip("torch")
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 40]


def _system(short):
    """A KKT system whose variables stand in LENGTHS constraints, then `short` variables in two each."""
    rng = np.random.default_rng(6)
    lengths = LENGTHS + [2] * short
    n, m = len(lengths), 41
    K = np.zeros((n + m, n + m))
    K[np.arange(n), np.arange(n)] = rng.uniform(0.5, 2.0, n)
    for j, k in enumerate(lengths):
        rows = n + rng.choice(m, k, replace=False)
        K[rows, j] = K[j, rows] = rng.standard_normal(k)
    K[np.arange(n, n + m), np.arange(n, n + m)] = -1e-2
    rows, cols = np.nonzero(K)
    rp = np.zeros(n + m + 1, np.int32)
    np.add.at(rp, rows + 1, 1)
    return np.cumsum(rp).astype(np.int32), cols.astype(np.int32), K[rows, cols], cb.kkt_blocking(n, m, 4)


@pytest.mark.parametrize("precision", [cb.F64, cb.F32])
@pytest.mark.parametrize("short", [0, 200])
def test_right_stage_exact(short, precision):
    dtype = np.float64 if precision == cb.F64 else np.float32
    rp, ci, v, bs = _system(short)
    n0, entries = len(LENGTHS) + short, sum(LENGTHS) + 2 * short
    assert (entries > 12 * n0) == (short == 0)  # one of each kind
    h = cb.Handle(0)
    F = cb.Factor(cb.Pattern(h, rp, ci, bs, 0, 1.0, precision))
    h.launch_count(reset=True)
    F.compute(torch.from_numpy(v.astype(dtype)).cuda())
    assert h.launch_count() == 3
    OF = oracle.Sym(rp, ci, bs, 0, 1.0, dtype).factor(v.astype(dtype))
    b = np.random.default_rng(5).standard_normal(len(rp) - 1).astype(dtype)
    want = OF.apply(cb.RIGHT, b)
    assert np.array_equal(F.apply(cb.RIGHT, torch.from_numpy(b).cuda()).cpu().numpy(), want)
    x = torch.from_numpy(b).cuda()
    F.apply(cb.RIGHT, x, x)
    assert np.array_equal(x.cpu().numpy(), want)
