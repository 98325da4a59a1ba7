"""The one-pass device quantiser where its strips, clusters and rounding can go wrong (needs a B200)."""
import ctypes

import pytest
import torch

import tensorrt_llm_b200 as pkg
from oracle import woq_oracle as o
from tensorrt_llm_b200 import quantize as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n,dtype,bits", [
    (64, 32, torch.float16, 8),        # one tile: a cluster of one; half a strip
    (448, 96, torch.bfloat16, 8),      # seven tiles: a cluster of four, the last CTA short
    (576, 64, torch.float32, 4),       # nine tiles on eight CTAs: some have none
    (4672, 192, torch.bfloat16, 4),    # narrow strips
    (4672, 96, torch.float32, 8),
    (9280, 64, torch.float16, 8),      # clusters of sixteen
    (9280, 64, torch.float32, 4),      # two passes
])
def test_strip_shapes(k, n, dtype, bits):
    torch.manual_seed(k + n)
    w = (torch.randn(k, n) * 0.02).to(dtype)
    w[:, 5] = 0          # a zero column
    w[:, 9] *= 1e-4      # (subnormal float16)
    if dtype != torch.float16:
        w[:, 11] *= 1e-33  # a scale too small for its reciprocal
    w[k // 2, 13] = -4 * w[:, 13].abs().max()
    u_ref, p_ref, s_ref = o.symmetric_quantize(w, bits)
    u, p, s = Q.symmetric_quantize_last_axis_of_batched_matrix_cuda(
        w.cuda(), torch.int8 if bits == 8 else torch.quint4x2, return_unprocessed=True)
    assert torch.equal(s.cpu().float(), s_ref.float())
    assert torch.equal(u.cpu(), u_ref)
    assert torch.equal(p.cpu(), p_ref)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("k,bits", [(576, 4), (576, 8), (4672, 4), (9280, 8)])
def test_not_a_number(k, bits, dtype):
    """A NaN quantises to 0 and does not count for its column's scale."""
    torch.manual_seed(k)
    w = (torch.randn(k, 64) * 0.02).to(dtype)
    nan = torch.zeros(k, 64, dtype=torch.bool)
    nan[torch.randint(0, k, (40,)), torch.randint(0, 48, (40,))] = True
    nan[:, 50] = True  # a whole column
    nan[3, 51] = True  # in a column of zeros
    w[:, 51] = 0
    u_ref, p_ref, s_ref = o.symmetric_quantize(w.masked_fill(nan, 0), bits)
    u, p, s = Q.symmetric_quantize_last_axis_of_batched_matrix_cuda(
        w.masked_fill(nan, float("nan")).cuda(), torch.int8 if bits == 8 else torch.quint4x2, return_unprocessed=True)
    assert torch.equal(s.cpu().float(), s_ref.float())
    assert torch.equal(u.cpu(), u_ref) and torch.equal(p.cpu(), p_ref)


def test_gemm_two_launches_behind_the_quantiser():
    """A layer whose weights were quantised before the preceding GEMM was enqueued may fetch them while that one
    runs: they have to be complete by then. (In a graph, so that launches follow each other closely; the last few
    columns are quantised when most of the chip has run empty.)"""
    k, n = 4096, 14336
    g = torch.Generator(device="cuda").manual_seed(1)
    ws = [(torch.randn(k, n, generator=g, device="cuda") * 0.02).bfloat16() for _ in range(3)]
    act = torch.randn(1, k, generator=g, device="cuda").bfloat16()
    other = Q.symmetric_quantize_last_axis_of_batched_matrix_cuda(ws[0][:, :64].contiguous(), torch.quint4x2)
    call = lambda p, s, out: pkg.ops.gemm_raw(act, p, s, out, n=out.numel(), k=k, weight_bits=4, group_size=0, weights_static=True)
    want = torch.empty(3, n, device="cuda", dtype=torch.bfloat16)
    for i, w in enumerate(ws):
        p, s = Q.symmetric_quantize_last_axis_of_batched_matrix_cuda(w, torch.quint4x2)
        torch.cuda.synchronize()
        call(p, s, want[i])
    lib, got = pkg._lib.lib(), torch.zeros(30, n, device="cuda", dtype=torch.bfloat16)
    scales, scales_t = torch.empty(n, device="cuda"), torch.empty(n, device="cuda", dtype=torch.bfloat16)
    processed, small = torch.empty_like(p), torch.empty(64, device="cuda", dtype=torch.bfloat16)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        for i in range(30):
            rc = lib.w4_symmetric_quantize_device(ptr(processed), None, ptr(scales), ptr(scales_t), pkg._lib.W4_DTYPE_BF16,
                                                  ptr(ws[i % 3]), pkg._lib.W4_DTYPE_BF16, k, n, 4, stream)
            assert rc == 0
            call(*other, small)
            call(processed, scales_t, got[i])
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(got[i], want[i % 3]) for i in range(30))
