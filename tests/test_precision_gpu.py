"""How close the outputs are to real arithmetic, beyond the bound of the oracle tests (needs a B200)."""
import pytest
import torch

import tensorrt_llm_b200 as pkg
from oracle import woq_oracle as oracle
from _cases import make_problem, max_err, oracle_out, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,bits,group,dtype", [
    (1, 14336, 4096, 8, 0, torch.float16),
    (4, 8192, 4096, 8, 128, torch.float16),
    (12, 4096, 4096, 4, 0, torch.bfloat16),
    (16, 4096, 4096, 4, 128, torch.bfloat16),
    (16, 8192, 2048, 8, 64, torch.float16),
])
def test_the_regime_decides_the_arithmetic(m, n, k, bits, group, dtype):
    """In the decode regime scales are applied to 32-bit sums, however the library would rather split the work:
    an automatic launch there is the requested decode launch bit for bit."""
    full = group != 0
    assert pkg.ops.select_regime(m, n, k, group, bits, dtype) == pkg.W4_REGIME_GEMV
    p = make_problem(m, n, k, bits, group, dtype, zero=full, bias=full, seed=m)
    assert torch.equal(run_gpu(p), run_gpu(p, regime=pkg.W4_REGIME_GEMV))


@pytest.mark.parametrize("bits,group,rows", [(4, 128, [3, 16, 40, 0, 9, 120]), (8, 0, [1, 1, 64, 5]), (8, 128, [2, 7])])
def test_experts_have_the_arithmetic_of_their_own_regime(bits, group, rows):
    n, k, dtype = 1024, 2048, torch.bfloat16
    first = [0]
    for r in rows:
        first.append(first[-1] + r)
    probs = [make_problem(max(r, 1), n, k, bits, group, dtype, zero=group != 0, seed=e) for e, r in enumerate(rows)]
    act = torch.cat([p["act"][:r] for p, r in zip(probs, rows)]).cuda()
    stack = lambda key: None if probs[0][key] is None else torch.stack([p[key] for p in probs]).cuda()
    out = pkg.ops.moe_gemm(act, stack("processed"), stack("scales"), first, weight_bits=bits, group_size=group,
                           zeros=stack("zeros")).cpu()
    regimes = set()
    for e, (p, r) in enumerate(zip(probs, rows)):
        if r == 0:
            continue
        got, regime = out[first[e]:first[e + 1]], pkg.ops.select_regime(r, n, k, group, bits, dtype)
        regimes.add(regime)
        if regime == pkg.W4_REGIME_GEMV:
            assert torch.equal(got, run_gpu(p, regime=regime)), e
        else:
            ref = oracle_out(p)
            assert max_err(got, ref) <= oracle.tolerance(ref), e
    assert pkg.W4_REGIME_GEMV in regimes
