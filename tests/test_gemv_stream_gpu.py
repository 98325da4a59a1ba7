"""The streaming decode kernel where its shares, tails and panels can go wrong (needs a B200)."""
import pytest
import torch

import tensorrt_llm_b200 as pkg
from oracle import woq_oracle as oracle
from _cases import make_problem, max_err, oracle_subset, run_gpu, sample_cols

pytestmark = pytest.mark.gpu


# every one of these sizes is in the streaming kernel's range: few rows and k units that leave the staged
# kernel's panels half empty, or many weights
@pytest.mark.parametrize("m,n,k,group,dtype", [
    (1, 8192, 2048, 128, torch.bfloat16),
    (2, 8384, 2176, 128, torch.float16),    # odd number of units, ragged column ranges
    (7, 8384, 2176, 0, torch.bfloat16),
    (8, 12352, 1152, 128, torch.bfloat16),
    (3, 9536, 4224, 128, torch.float16),    # one unit more than the staged kernel's panel
    (5, 24640, 128, 0, torch.bfloat16),     # a single unit: most warps have no share of a column group
    (6, 16384, 20480, 128, torch.bfloat16),  # two activation panels
])
def test_shares_tails_and_panels(m, n, k, group, dtype):
    full = group != 0
    p = make_problem(m, n, k, 4, group, dtype, zero=full, bias=full, prequant=full, seed=m + k)
    if dtype == torch.bfloat16:  # values far outside float16's range, and zeros
        p["act"][0] *= 2.0 ** 40
        p["act"][-1, :130] = 0
        if m > 1:
            p["act"][1] *= 2.0 ** -60
    alpha = 0.5 if full else 1.0
    out = run_gpu(p, regime=pkg.W4_REGIME_GEMV, alpha=alpha)
    cols = sample_cols(n, count=64)
    for row in range(m):
        ref = oracle_subset(p, [row], cols, alpha=alpha)
        assert max_err(out[[row]][:, cols], ref) <= oracle.tolerance(ref), row
    assert torch.equal(out, run_gpu(p, regime=pkg.W4_REGIME_GEMV, alpha=alpha))  # sums in a fixed order
    assert pkg._lib.lib().w4_gemm_device_status() == 0


@pytest.mark.parametrize("n,k", [(8192, 2048), (1024, 1024)])  # streaming kernel, staged kernel
def test_activations_written_by_the_kernel_in_front(n, k):
    """The kernels are resident while the kernel in front still writes their activations: what they read is what it
    wrote last. (A read past that rule need not show here; the loads are ordinary ones for that reason.)"""
    p = make_problem(2, n, k, 4, 128, torch.bfloat16, zero=True, prequant=True, seed=k)
    w, s, z, ps = (p[key].cuda() for key in ("processed", "scales", "zeros", "ps"))
    call = lambda a: pkg.ops.weight_only_groupwise_quant_matmul(a, ps, w, s, z, None, 1.0, pkg.ZERO | pkg.PRE_QUANT_SCALE, 128,
                                                                weights_static=True)
    acts = [torch.randn(2, k, generator=torch.Generator().manual_seed(i)).bfloat16().cuda() for i in range(8)]
    want = [call(a) for a in acts]
    buf, got = torch.empty_like(acts[0]), []
    for i in range(200):
        buf.copy_(acts[i % 8])
        got.append(call(buf))
    assert all(torch.equal(got[i], want[i % 8]) for i in range(200))


def test_one_row_is_not_slower_than_eight():
    """The weights are the same and the activations fewer. (With the wrong split of L1 and shared memory, which
    depended on the activations' size, one row took 80 us here and eight 54.)"""
    n, k = 57344, 8192
    w = torch.randint(-128, 128, (k, n // 2), dtype=torch.int8, device="cuda")
    s, z = (torch.rand(k // 128, n, device="cuda").bfloat16() for _ in range(2))

    def us(m):
        a, out = torch.randn(m, k, device="cuda").bfloat16(), torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
        call = lambda: pkg.ops.gemm_raw(a, w, s, out, n=n, k=k, weight_bits=4, group_size=128, zeros=z,
                                        regime=pkg.W4_REGIME_GEMV, weights_static=True)
        best = 1e9
        for _ in range(8):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            call()
            e0.record()
            for _ in range(20):
                call()
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1) * 50)
        return best

    one, eight = us(1), us(8)
    assert one < 1.15 * eight
