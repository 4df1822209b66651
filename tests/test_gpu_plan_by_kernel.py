"""The decode plan a component uploads follows the kernel its profile takes: equal pieces only where a CTA's warps take a tile
each; the CUDA-core kernels keep the equal shares that psi_plan_preview lays out, whatever mode they were reached by."""
import numpy as np
import pytest

import decode_preview as P
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


@pytest.mark.parametrize("dtype,heads,head_dim,page", [(pkg.BF16, (40, 8), 128, 8), (pkg.F16, (16, 4), 64, 16), (pkg.BF16, (24, 8), 96, 12), (pkg.BF16, (16, 2), 200, 16),
                                                       (pkg.F32, (16, 2), 256, 16), (pkg.F32, (8, 2), 80, 16), (pkg.BF16, (4, 2), 66, 16)])
@pytest.mark.parametrize("contexts", [[300], [777, 3], [370] * 8, [1000, 40, 9000]])
def test_the_preview_is_what_prepare_uploads(dtype, heads, head_dim, page, contexts):
    s = W.Session(W.Spec("plan", dtype, *heads, head_dim, page, contexts, [1] * len(contexts), seed=95), max_ctas=100)
    stats = s.gqa.plan_stats()
    s.close()
    counts = P.preview(P.config(dtype, heads, head_dim, page, pkg.KERNEL_AUTO), contexts, np.arange(len(contexts) + 1), 100)[2]
    assert tuple(int(x) for x in counts) == tuple(stats[k] for k in ("items", "ctas", "partial_slots", "reduce_units", "q_tiles", "kv_tiles"))
