"""The decode plan a component uploads follows the kernel its profile takes: equal pieces only where a CTA's warps take a tile
each; the CUDA-core kernels keep the equal shares that psi_plan_preview lays out, whatever mode they were reached by."""
import numpy as np
import pytest

import gpuharness as G
import hostapi as H
import workloads as W

pkg = G.pkg
pytestmark = pytest.mark.gpu

STEPS = {"one": ((40, 8), [300]), "eight": ((16, 2), [370] * 8), "ragged": ((16, 2), [1, 40, 800, 90, 17])}


def _plans(dtype, step, head_dim, mode, min_tiles, start_cost):
    heads, contexts = STEPS[step]
    s = W.Session(W.Spec("plan", dtype, *heads, head_dim, 16, contexts, [1] * len(contexts), seed=95), kernel_mode=mode, max_ctas=296)
    stats = s.gqa.plan_stats()
    s.close()
    counts = H.plan_preview(*heads, np.asarray(contexts), np.arange(len(contexts) + 1), 296, min_tiles, start_cost)[2]
    return (stats["items"], stats["ctas"], stats["partial_slots"], stats["reduce_units"]), tuple(int(x) for x in counts[:4])


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("dtype,head_dim,mode", [(pkg.F32, 80, pkg.KERNEL_AUTO), (pkg.F32, 6, pkg.KERNEL_AUTO), (pkg.BF16, 84, pkg.KERNEL_AUTO),
                                                 (pkg.BF16, 66, pkg.KERNEL_AUTO), (pkg.F16, 33, pkg.KERNEL_AUTO), (pkg.F32, 128, pkg.KERNEL_GENERIC),
                                                 (pkg.BF16, 128, pkg.KERNEL_GENERIC), (pkg.BF16, 96, pkg.KERNEL_GENERIC)])
def test_the_cuda_core_kernels_keep_the_shares(dtype, head_dim, mode, step):
    uploaded, shares = _plans(dtype, step, head_dim, mode, 4, 0)
    assert uploaded == shares


@pytest.mark.parametrize("dtype,head_dim,min_tiles,start_cost", [(pkg.BF16, 128, 16, 32), (pkg.F16, 64, 16, 32), (pkg.BF16, 96, 4, 16), (pkg.F32, 128, 4, 0)])
def test_the_other_kernels_take_pieces(dtype, head_dim, min_tiles, start_cost):
    # 64 units of 300 tokens: a start each in the shares, a CTA each in the pieces
    heads, contexts = (16, 2), [300] * 32
    s = W.Session(W.Spec("plan", dtype, *heads, head_dim, 16, contexts, [1] * 32, seed=95))
    stats = s.gqa.plan_stats()
    s.close()
    assert stats["items"] == stats["ctas"] >= 64
