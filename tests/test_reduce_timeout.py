"""The bounded wait of the persistent solver's reductions.

A fused two-level iteration with short rows counts its reductions' barrier on
a device counter and waits at most 200 ms; culipx_sqmr_set_reduce_skew raises
the count beyond reach, so the wait gives up, every CTA leaves the loop and the
solve ends in CULIPX_TIMEOUT.  Every other solve -- level loops with grid
barriers of their own, or a row long enough for a phase to come near the limit
-- keeps an unbounded grid barrier, which the skew does not touch."""
import numpy as np
import pytest

import culip_b200 as cb
from culip_b200 import _capi as capi
from problems import kkt, scrambled_kkt

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
sp = pytest.importorskip("scipy.sparse")

SKEW = 1 << 40


def _with_dense_row(n, m=64):
    """A KKT system whose first constraint has all n variables: its row of K has n + 1 entries."""
    rng = np.random.default_rng(5)
    A = sp.random(m, n, density=0.002, random_state=5, format="lil")
    A[0] = rng.uniform(0.5, 1.5, n)
    H = sp.diags(rng.uniform(0.5, 2.0, n))
    K = sp.bmat([[H, A.T], [A, -1e-2 * sp.identity(m)]], format="csr")
    K.sort_indices()
    return K.indptr.astype(np.int32), K.indices.astype(np.int32), K.data, cb.kkt_blocking(n, m, 8)


def _setup(h, system, precision=cb.F64):
    rp, ci, v, bs = system
    F = cb.Factor(cb.Pattern(h, rp, ci, bs, 0, 1.0, precision))
    F.compute(torch.from_numpy(v).cuda().to(torch.float64 if precision == cb.F64 else torch.float32))
    A = cb.CsrOperator(h, torch.from_numpy(rp).cuda(), torch.from_numpy(ci).cuda(), torch.from_numpy(v).cuda())
    return F, A, torch.from_numpy(cb.normal_vector(cb.SEED + 1, len(rp) - 1)).cuda()


def _skew(h, value):
    capi.call("culipx_sqmr_set_reduce_skew", h._h, value)


@pytest.mark.parametrize("system", ["small", "row of 8192"])
def test_counted_reduction_times_out_and_the_handle_recovers(system):
    h = cb.Handle(0)
    F, A, b = _setup(h, kkt("small") if system == "small" else _with_dense_row(8191))
    x_ref = torch.zeros_like(b)
    ref = cb.sqmr_solve(h, A, F, b, x_ref, 1e-8, 12)
    _skew(h, SKEW)
    with pytest.raises(cb.CulipxError) as err:
        cb.sqmr_solve(h, A, F, b, torch.zeros_like(b), 1e-8, 100000)
    assert err.value.status == capi.TIMEOUT
    B = torch.stack([b, 2.0 * b, -b])
    assert np.all(cb.sqmr_solve_multi(h, A, F, B, torch.zeros_like(B), 1e-8, 100000)[2] == capi.TIMEOUT)
    _skew(h, 0)
    x = torch.zeros_like(b)
    assert cb.sqmr_solve(h, A, F, b, x, 1e-8, 12) == ref
    assert torch.equal(x, x_ref)


@pytest.mark.parametrize("system", ["deep levels", "row of 8193", "row of 20001"])
def test_unbounded_where_a_phase_may_be_long(system):
    h = cb.Handle(0)
    F, A, b = _setup(h, scrambled_kkt() if system == "deep levels" else _with_dense_row(int(system[7:]) - 1))
    B = torch.stack([b, 2.0 * b, -b, 0.5 * b])
    x_ref, X_ref = torch.zeros_like(b), torch.zeros_like(B)
    ref = cb.sqmr_solve(h, A, F, b, x_ref, 1e-12, 12)
    ref_multi = cb.sqmr_solve_multi(h, A, F, B, X_ref, 1e-12, 12)
    _skew(h, SKEW)
    x, X = torch.zeros_like(b), torch.zeros_like(B)
    assert cb.sqmr_solve(h, A, F, b, x, 1e-12, 12) == ref
    multi = cb.sqmr_solve_multi(h, A, F, B, X, 1e-12, 12)
    _skew(h, 0)
    assert all(np.array_equal(got, want) for got, want in zip(multi, ref_multi))
    assert torch.equal(x, x_ref) and torch.equal(X, X_ref)
