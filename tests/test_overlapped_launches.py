"""Kernels that are launched over their predecessor's end (csrc/launch.cuh).

Their life begins before the predecessor has finished writing.  Each has to
wait (wait_previous, after_previous), and what the predecessor may have written has to be read
with ordinary loads: neither __ldg nor a const __restrict__ parameter, which
promise memory that nothing writes during the kernel's life.  The sources are
checked here; on the GPU, chains of dependent calls without a host
synchronisation must give the bits of the same calls one at a time."""
import os
import re

import numpy as np
import pytest

import culip_b200 as cb

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "culip_b200", "csrc")

# what the kernel before may write, per source and function
WRITTEN = {
    "spmv.cu": {"k_csr_spmv": ["val", "x", "y"], "k_csr_spmv_rows": ["val", "x", "y"], "k_sell_spmv": ["x", "y"],
                "k_long_rows": ["x", "y"]},
    "kkt_assembly.cu": {"k_kkt_values": ["aval", "x", "s", "d", "kval"]},
    "solve.cu": {"k_solve_D": ["in", "out"]},
    "factor_two_level.cu": {"level0_pivot": ["kval"], "k_two_rows": ["kval"], "spread_nonfinite": ["up", "dg"],
                            "k_two_tiles": ["up", "nonfinite"],
                            "split_rows": ["kind", "kinds", "rowflags", "ndmask"], "k_two_order": ["up", "iperm"]},
    "apply_two_level.cu": {"k_two_left": ["b", "x"], "k_two_right_tiles": ["b", "x"], "k_two_right_rows": ["b", "x"]},
}


def _function(source, name):
    """(parameters, body) of a function of a source."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, source)).read())
    for start in (m.end() for m in re.finditer(rf"\b{name}\(", text)):
        close = _closing(text, start, "()")
        rest = text[close + 1:].lstrip()
        if rest.startswith("{"):
            body = text.index("{", close) + 1
            return text[start:close], text[body:_closing(text, body, "{}")]
    raise AssertionError(f"{source} defines no {name}")


def _closing(text, at, pair):
    """Where the bracket that was opened just before `at` closes."""
    depth = 1
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[at], 0)
        if depth == 0:
            return at
        at += 1


def _overlapped_sources():
    return [f for f in sorted(os.listdir(CSRC)) if f.endswith(".cu")
            and "launch_overlapped(" in open(os.path.join(CSRC, f)).read()]


def test_every_overlapped_kernel_waits():
    assert set(_overlapped_sources()) == set(WRITTEN)
    for source in WRITTEN:
        text = open(os.path.join(CSRC, source)).read()
        launched = set(re.findall(r"launch_overlapped\(\s*(\w+)<", text))
        assert launched
        for kernel in launched:
            assert re.search(r"(after|wait)_previous\(\)", _function(source, kernel)[1]), kernel
            assert kernel in WRITTEN[source], kernel


@pytest.mark.parametrize("source", sorted(WRITTEN))
def test_a_predecessors_output_is_read_with_ordinary_loads(source):
    for name, buffers in WRITTEN[source].items():
        parameters, body = _function(source, name)
        for v in buffers:
            assert not re.search(rf"__restrict__\s+{v}\b", parameters), (name, v)
            assert not re.search(rf"__ld\w+\(\s*&?(a\.)?{v}\b", body), (name, v)


# ---------------------------------------------------------------------------
# on the GPU


def _program(precision):
    """Everything a step of an interior-point program holds, on one stream."""
    torch = pytest.importorskip("torch")
    h = cb.Handle(0)
    n, m = 4001, 1999
    rp, ci, v = cb.kkt_generate(n, m, 5, 32, 1e-2, 1e2, seed=9)
    first = int(rp[n])
    keep = np.ones(len(ci) - first, bool)
    keep[rp[n + 1:] - 1 - first] = False
    arp = (rp[n:] - first - np.arange(m + 1)).astype(np.int32)
    aci, av = ci[first:][keep].astype(np.int32), v[first:][keep].astype(np.float64)
    dtype = torch.float64 if precision == cb.F64 else torch.float32
    d = [torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (arp, aci, av)]
    asm = cb.KktAssembly(h, m, n, d[0], d[1])
    krp, kci = asm.structure()
    kval = torch.empty(asm.nnz, dtype=dtype, device="cuda")
    F = cb.Factor(cb.Pattern(h, krp, kci, cb.kkt_blocking(n, m, 8), 0, 1.0, precision))
    A = cb.CsrOperator(h, torch.from_numpy(krp).cuda(), torch.from_numpy(kci).cuda(), kval)  # borrows kval
    return dict(torch=torch, h=h, n=n, N=n + m, aval=d[2], asm=asm, kval=kval, F=F, A=A, dtype=dtype)


def _step(p, x, s, b, wait):
    """Assembly -> factor -> stages -> products; every call reads the one before."""
    torch, N, dtype = p["torch"], p["N"], p["dtype"]
    t = [torch.zeros(N, dtype=dtype, device="cuda") for _ in range(6)]

    def then(result):
        if wait:
            torch.cuda.synchronize()
        return result

    then(p["asm"].assemble(p["aval"], p["kval"], x=x, s=s, delta=1e-6, gamma=1e-6))
    then(p["A"].spmv(b, t[0]))                       # K's values straight from the assembly
    then(p["A"].spmv(t[0], t[1]))                    # the product of a product
    then(p["A"].spmv(t[1], t[0], alpha=-0.5, beta=0.25))  # back into the first, its values in use
    then(p["asm"].assemble(p["aval"], p["kval"], x=x, s=s, delta=2e-6, gamma=1e-6))
    then(p["F"].compute(p["kval"]))                  # the factor straight from the assembly
    then(p["F"].apply(cb.LEFT, b, t[2]))
    then(p["F"].apply(cb.MIDDLE, t[2], t[3]))
    then(p["F"].apply(cb.RIGHT, t[3], t[4]))
    then(p["A"].spmv(t[4], t[5]))
    then(p["F"].apply(cb.MIDDLE, t[5], t[5]))        # in place, on the product's output
    return t


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [cb.F64, cb.F32])
def test_dependent_calls_without_synchronisation(precision):
    p = _program(precision)
    torch = p["torch"]
    g = torch.Generator(device="cuda").manual_seed(3)
    inputs = []
    for _ in range(24):  # other values each time, spread so that the tiles' swaps differ
        x = torch.exp(torch.randn(p["n"], generator=g, device="cuda", dtype=torch.float64))
        s = x * torch.exp(3 * torch.randn(p["n"], generator=g, device="cuda", dtype=torch.float64))
        inputs.append((x, s, torch.randn(p["N"], generator=g, device="cuda", dtype=torch.float64).to(p["dtype"])))
    torch.cuda.synchronize()
    chained = [_step(p, *i, wait=False) for i in inputs]
    torch.cuda.synchronize()
    one_at_a_time = [_step(p, *i, wait=True) for i in inputs]
    for k, (got, want) in enumerate(zip(chained, one_at_a_time)):
        for j in range(6):
            assert torch.equal(got[j], want[j]), (k, j)
