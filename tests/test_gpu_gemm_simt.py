"""The 32-bit matrix products: every kernel of the file against float64, and the promise that an output has the same bits whichever
kernel takes its row (few rows, large tiles, small tiles, blocks of K over a cluster, rows on no 16-byte boundary)."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


# K: below, at and above blocks of 512, spans of 2,048 and chunks of 32 and 64 at a span's end; one block over 16 (no cluster); N: remainders of 8, 32 and 128
@pytest.mark.parametrize("n,k", [(7, 4), (100, 172), (130, 512), (129, 516), (260, 2048), (65, 2052), (2100, 1028), (70, 8704),
                                 (70, 32), (33, 36), (64, 64), (40, 68), (24, 500), (24, 2080), (9, 6212)])
def test_outputs_do_not_depend_on_the_kernel(n, k):
    from kuiperllama_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(n * k)
    a = torch.randn(1100, k, device=DEV, generator=g)
    w = torch.randn(n, k, device=DEV, generator=g)
    exact = a.double() @ w.double().T
    # a chain of 512 and a sum of k / 512 blocks: each addition is off by half a unit of a partial sum below |a||w|
    bound = (512 + k / 512 + 2) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    whole = torch.empty(1100, n, device=DEV)
    ops.gemm_simt(a, w, whole)
    assert bool(((whole.double() - exact).abs() <= bound).all())
    odd = torch.zeros(1100, k + 1, device=DEV)                  # the same rows at a stride that no 16-byte copy takes
    odd[:, :k] = a
    for m in (1, 2, 3, 8, 9, 16, 17, 64, 65, 333):
        for rows in (a[:m], odd[:m, :k]):
            out = torch.full((m + 1, n), 5.0, device=DEV)
            ops.gemm_simt(rows, w, out[:m])
            assert torch.equal(out[:m], whole[:m]), f"{m} rows"
            assert bool((out[m] == 5.0).all())


# steps of 16 columns in groups of four (small tiles) or one by one (large ones): below a step, at and past a group and two groups
@pytest.mark.parametrize("n,k", [(5, 3), (33, 16), (40, 60), (64, 64), (31, 66), (96, 172), (130, 1030), (40, 2051)])
def test_bfloat16_operands_give_the_bits_of_their_float32_copies(n, k):
    from kuiperllama_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(n * k)
    a, w = torch.randn(4100, k, device=DEV, generator=g).bfloat16(), torch.randn(n, k, device=DEV, generator=g).bfloat16()
    for m in (1, 9, 64, 65, 4100):                              # small tiles, and (130 features) large ones
        want, got = torch.empty(m, n, device=DEV), torch.full((m + 1, n), 5.0, device=DEV)
        ops.gemm_simt(a[:m].float(), w.float(), want)
        ops.gemm_simt(a[:m], w, got[:m])
        assert torch.equal(got[:m], want) and bool((got[m] == 5.0).all()), m
        rounded = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
        ops.gemm_simt(a[:m], w, rounded)
        assert torch.equal(rounded, want.bfloat16()), m
