"""psi_decode_plan_preview: the shares of psi_plan_preview where a profile's kernel keeps them, equal pieces of one CTA each where
it takes them (no GPU)."""
import numpy as np
import pytest

import decode_preview as P
import hostapi as H

pkg = P.pkg


@pytest.mark.parametrize("dtype,head_dim,mode", [(pkg.F32, 80, pkg.KERNEL_AUTO), (pkg.BF16, 66, pkg.KERNEL_AUTO), (pkg.BF16, 128, pkg.KERNEL_GENERIC)])
@pytest.mark.parametrize("heads,contexts", [((40, 8), [300]), ((16, 2), [370] * 8), ((16, 2), [1, 40, 800])])
def test_cuda_core_profiles_get_the_shares(dtype, head_dim, mode, heads, contexts):
    cu = np.arange(len(contexts) + 1)
    got = P.preview(P.config(dtype, heads, head_dim, 16, mode), contexts, cu, 296)
    shares = H.plan_preview(*heads, np.asarray(contexts), cu, 296, 4, 0)
    for a, b in zip(got, shares):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dtype,heads,head_dim,contexts", [(pkg.BF16, (40, 8), 128, [777]), (pkg.F16, (16, 4), 64, [300] * 8), (pkg.BF16, (24, 8), 96, [1000] * 16),
                                                           (pkg.F32, (16, 2), 256, [300] * 16), (pkg.BF16, (16, 2), 200, [600] * 16)])
def test_small_steps_get_pieces(dtype, heads, head_dim, contexts):
    items, ctas, counts = P.preview(P.config(dtype, heads, head_dim, 16, pkg.KERNEL_AUTO), contexts, np.arange(len(contexts) + 1), 148)
    assert np.array_equal(ctas, np.arange(len(items) + 1)) and int(counts[1]) <= 148
    length = {}
    for tile, head, begin, end, _, _ in items.tolist():
        assert begin == length.get((tile, head), 0)
        length[tile, head] = end
    assert sorted(length) == [(t, h) for t in range(len(contexts)) for h in range(heads[1])]
    assert all(length[t, h] == contexts[t] + 1 for t, h in length)
    tiles = -(-(items[:, 3].astype(int) - items[:, 2]) // 16)
    assert tiles.max() - tiles.min() <= 1


def test_a_long_step_keeps_the_shares():
    contexts = np.linspace(1024, 8192, 32).astype(int)
    got = P.preview(P.config(pkg.BF16, (16, 2), 256, 16, pkg.KERNEL_AUTO), contexts, np.arange(33), 148)
    for a, b in zip(got, H.plan_preview(16, 2, contexts, np.arange(33), 148, 16, 32)):
        assert np.array_equal(a, b)


def test_what_prepare_would_refuse_is_refused():
    ti, cu, counts = np.array([5], dtype=np.uint32), np.array([0, 1], dtype=np.uint32), np.zeros(6, dtype=np.uint32)
    for cfg in (P.config(pkg.F32, (16, 2), 128, 16, pkg.KERNEL_MMA), P.config(pkg.BF16, (16, 3), 128, 16, pkg.KERNEL_AUTO), P.config(pkg.BF16, (16, 2), 264, 16, pkg.KERNEL_AUTO),
                P.config(7, (16, 2), 128, 16, pkg.KERNEL_AUTO)):
        assert P.status_of(cfg, ti, cu, 148, None, None, counts) != 0
    cfg = P.config(pkg.BF16, (16, 2), 128, 16, pkg.KERNEL_AUTO)
    assert P.status_of(cfg, ti, cu, 148, None, None, counts) == 0
    assert P.status_of(cfg, ti, np.array([1, 2], dtype=np.uint32), 148, None, None, counts) != 0
    assert P.status_of(cfg, ti, cu, 148, np.zeros((1, 6), dtype=np.uint32), None, counts) != 0  # (two units)
