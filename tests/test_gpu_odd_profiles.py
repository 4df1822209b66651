"""The tensor-core kernel for 16-bit profiles off the beaten track: head sizes around its padded widths, pages that are no
power of two, row counts up to a full tile; and its precision, which is that of the CUDA-core kernel."""
import numpy as np
import pytest

import checks
import workloads as W
import gpuharness as G
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [pkg.BF16, pkg.F16])
@pytest.mark.parametrize("heads,runs", [((3, 1), [1, 1, 1, 1]), ((24, 8), [1, 2, 1, 5]), ((17, 1), [1, 1, 1, 1])])
@pytest.mark.parametrize("head_dim,page", [(8, 1), (64, 12), (72, 16), (80, 16), (96, 12), (128, 5), (136, 16), (192, 7), (200, 8), (256, 24)])
def test_odd_profiles_match_the_oracle(dtype, heads, runs, head_dim, page):
    spec = W.Spec("odd", dtype, *heads, head_dim, page, [1, 15, 1037, 2600], runs, seed=5)
    s = W.Session(spec)
    s.append()
    s.attend()
    s.ctx.sync()
    checks.assert_attention_close(s)
    s.close()


@pytest.mark.parametrize("dtype", [pkg.BF16, pkg.F16])
@pytest.mark.parametrize("head_dim", [96, 200])
def test_partials_keep_f32_precision(dtype, head_dim):
    # weights in f32: the partial outputs are as close to the f32 oracle as the CUDA-core kernel's
    import torch
    worst = {}
    for mode in (pkg.KERNEL_AUTO, pkg.KERNEL_GENERIC):
        s = W.Session(W.Spec("odd", dtype, 8, 2, head_dim, 12, [40, 9000], [1, 1], seed=6), kernel_mode=mode)
        o, m, l = torch.zeros(s.q.shape, device=s.device), torch.zeros(s.q.shape[:2], device=s.device), torch.zeros(s.q.shape[:2], device=s.device)
        s.append()
        s.gqa.attend_partial(s.pages, s.table, 0, s.q, o, m, l)
        s.ctx.sync()
        expected, rows = checks.oracle_attention(s)
        worst[mode] = np.abs(checks.to_numpy_bits(o)[rows] - expected).max()
        s.close()
    assert worst[pkg.KERNEL_AUTO] <= max(2e-6, 2 * worst[pkg.KERNEL_GENERIC]), worst


def test_unaligned_buffers_keep_the_cuda_core_kernel():
    import torch
    s = W.Session(W.Spec("odd", pkg.BF16, 6, 2, 96, 12, [500, 70], [1, 2], seed=7))
    s.append()
    out = torch.zeros(s.q.numel() + 1, dtype=s.tdtype, device=s.device)[1:].view(s.q.shape)
    s.gqa.attend(s.pages, s.table, 0, s.q, out)
    s.gqa.attend(s.pages, s.table, 0, s.q, s.out)
    s.ctx.sync()
    a, b = (O.decode(checks.to_numpy_bits(x), pkg.BF16) for x in (out, s.out))
    assert np.abs(a - b).max() <= 2e-2
    checks.assert_attention_close(s)
    s.close()
