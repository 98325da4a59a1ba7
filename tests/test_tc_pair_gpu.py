"""The CTA-pair tensor-core kernel at the sizes where its tiles, rings and splits can go wrong (needs a B200)."""
import ctypes

import pytest
import torch

import tensorrt_llm_b200 as pkg
from tensorrt_llm_b200._lib import W4GemmParams
from oracle import woq_oracle as oracle
from _cases import make_problem, max_err, oracle_out, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,bits,group,dtype", [
    (31, 64, 64, 4, 64, torch.bfloat16),      # one half-filled step; the pair's second CTA has no columns
    (33, 320, 128, 4, 128, torch.float16),    # the second pair tile has half of one CTA's columns
    (257, 192, 192, 8, 64, torch.bfloat16),   # two row tiles, odd number of 64-k halves
    (160, 8192, 1152, 8, 0, torch.bfloat16),  # seven weight stages, nine steps, three conversion groups
    (224, 16640, 832, 4, 64, torch.float16),  # single accumulator, rings that wrap at different places
    (96, 19200, 640, 8, 128, torch.float16),  # two accumulators, more tiles than pairs
    (64, 1280, 2048, 4, 128, torch.bfloat16),  # splits that share a cluster
    (17, 96, 8192, 8, 0, torch.float16),      # one tile, the largest cluster
    (250, 512, 4096, 4, 64, torch.bfloat16),  # cluster splits of a 256-row tile
    (40, 256, 4224, 4, 128, torch.bfloat16),  # 33 steps: the last split is shorter
])
def test_tile_ring_and_split_edges(m, n, k, bits, group, dtype):
    full = group != 0
    p = make_problem(m, n, k, bits, group, dtype, zero=full, bias=full, seed=m + n)
    alpha = 0.5 if full else 1.0
    rows = sorted({0, m - 1, *range(0, m, 29)})
    for _ in range(3):  # back to back: the next launch's weights are fetched while the previous one drains
        out = run_gpu(p, regime=pkg.W4_REGIME_GEMM, alpha=alpha)
    ref = oracle_out(dict(p, act=p["act"][rows].contiguous(), m=len(rows)), alpha=alpha)
    assert max_err(out[rows], ref) <= oracle.tolerance(ref)
    assert torch.equal(out, run_gpu(p, regime=pkg.W4_REGIME_GEMM, alpha=alpha))  # sums in a fixed order
    assert pkg._lib.lib().w4_gemm_device_status() == 0


@pytest.mark.parametrize("m,n,k,bits", [(9, 14336, 1024, 4), (16, 4096, 4096, 4), (12, 8192, 2048, 8)])
def test_decode_regime_through_the_tensor_cores(m, n, k, bits):
    """9 to 16 rows in the decode regime: whichever kernel the launch takes needs no workspace and agrees
    with the decode kernel to rounding."""
    p = make_problem(m, n, k, bits, 128, torch.bfloat16, zero=True, bias=True, seed=m)
    assert pkg.ops.workspace_bytes(m, n, k, 128, bits, torch.bfloat16, False) == 0
    auto, decode = run_gpu(p), run_gpu(p, regime=pkg.W4_REGIME_GEMV)
    ref = oracle_out(p)
    assert max_err(auto, ref) <= oracle.tolerance(ref) and max_err(auto, decode) <= oracle.tolerance(ref)


@pytest.mark.parametrize("bits,group,rows,k,n", [
    (4, 128, [1] * 40, 256, 320),                # more experts than one launch holds; a pair tile half empty
    (8, 0, [0, 33, 0, 1, 64, 300, 0], 576, 96),  # experts without rows, several row tiles, an odd half step
    (4, 64, [5, 6], 4096, 256),                  # few tiles: cluster splits
])
def test_experts_in_one_launch(bits, group, rows, k, n):
    full = group != 0
    first = [0]
    for r in rows:
        first.append(first[-1] + r)
    probs = [make_problem(max(r, 1), n, k, bits, group, torch.bfloat16, zero=full, bias=full, seed=e)
             for e, r in enumerate(rows)]
    act = torch.cat([p["act"][:r] for p, r in zip(probs, rows)]).cuda()
    stack = lambda key: None if probs[0][key] is None else torch.stack([p[key] for p in probs]).cuda()
    out = pkg.ops.moe_gemm(act, stack("processed"), stack("scales"), first, weight_bits=bits, group_size=group,
                           zeros=stack("zeros"), bias=stack("bias"), alpha=0.5 if full else 1.0).cpu()
    for e, (p, r) in enumerate(zip(probs, rows)):
        if r:
            ref = oracle_out(dict(p, act=p["act"][:r]), alpha=0.5 if full else 1.0)
            assert max_err(out[first[e]:first[e + 1]], ref) <= oracle.tolerance(ref), e
    assert pkg._lib.lib().w4_gemm_device_status() == 0


def test_last_expert_of_a_launch_keeps_to_its_own_rows():
    """33 experts are a launch of 32 and one of a single expert; given a workspace, that one must not use the
    split that adds up and stores the whole output (a few tiles and a long k, where its plan would). Through the
    C ABI, where callers pass a workspace."""
    experts, rows, n, k = 33, 33, 64, 16384
    assert pkg.ops.select_regime(rows, n, k, 64, 4, torch.bfloat16) == pkg.W4_REGIME_GEMM
    first = [rows * e for e in range(experts + 1)]
    probs = [make_problem(rows, n, k, 4, 64, torch.bfloat16, zero=True, bias=True, seed=e) for e in range(experts)]
    act = torch.cat([p["act"] for p in probs]).cuda()
    weight, scales, zeros, bias = (torch.stack([p[key] for p in probs]).cuda()
                                   for key in ("processed", "scales", "zeros", "bias"))
    out = torch.empty((experts * rows, n), dtype=torch.bfloat16, device="cuda")
    ws = torch.zeros(64 << 20, dtype=torch.uint8, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    params = W4GemmParams(act=ptr(act), weight=ptr(weight), scales=ptr(scales), zeros=ptr(zeros), bias=ptr(bias),
                          out=ptr(out), alpha=0.5, m=experts * rows, n=n, k=k, group_size=64, weight_bits=4,
                          act_dtype=pkg._lib.W4_DTYPE_BF16, workspace=ptr(ws), workspace_bytes=ws.numel())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = pkg._lib.lib().w4_gemm_launch_experts(ctypes.byref(params), experts, (ctypes.c_int * len(first))(*first), stream)
    assert rc == 0
    got = out.cpu()
    for e, p in enumerate(probs):
        ref = oracle_out(p, alpha=0.5)
        assert max_err(got[first[e]:first[e + 1]], ref) <= oracle.tolerance(ref), e
    assert pkg._lib.lib().w4_gemm_device_status() == 0
