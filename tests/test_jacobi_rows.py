"""Block-Jacobi sweeps (SOLVE_JACOBI) over rows on both sides of a batch of
loads, in block rows with and without a pivot tile to substitute with: the
oracle's sweeps, bit for bit."""
import numpy as np
import pytest

import culip_b200 as cb

torch = pytest.importorskip("torch")
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _system(lengths, n):
    """A KKT system whose constraint rows have the given numbers of entries."""
    rng = np.random.default_rng(4)
    m = len(lengths)
    K = np.zeros((n + m, n + m))
    K[np.arange(n), np.arange(n)] = rng.uniform(0.5, 2.0, n)
    for i, k in enumerate(lengths):
        cols = rng.choice(n, k, replace=False)
        K[n + i, cols] = K[cols, n + i] = rng.standard_normal(k)
    K[np.arange(n, n + m), np.arange(n, n + m)] = -1e-2
    rows, cols = np.nonzero(K)
    rp = np.zeros(n + m + 1, np.int32)
    np.add.at(rp, rows + 1, 1)
    return np.cumsum(rp).astype(np.int32), cols.astype(np.int32), K[rows, cols]


@pytest.mark.parametrize("precision", [cb.F64, cb.F32])
@pytest.mark.parametrize("block", [1, 8, 32])
def test_jacobi_sweeps_exact(block, precision):
    dtype = np.float64 if precision == cb.F64 else np.float32
    lengths = [1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 49, 100]
    rp, ci, v = _system(lengths, 101)
    bs = cb.kkt_blocking(101, len(lengths), block)
    F = cb.Factor(cb.Pattern(cb.Handle(0), rp, ci, bs, 0, 1.0, precision))
    F.compute(torch.from_numpy(v.astype(dtype)).cuda())
    OF = oracle.Sym(rp, ci, bs, 0, 1.0, dtype).factor(v.astype(dtype))
    b = np.random.default_rng(5).standard_normal(len(rp) - 1).astype(dtype)
    F.set_solve_algorithm(cb.SOLVE_JACOBI, 3)
    for stage in (cb.LEFT, cb.RIGHT):
        got = F.apply(stage, torch.from_numpy(b).cuda()).cpu().numpy()
        assert np.array_equal(got, OF.apply(stage, b, 3)), stage
