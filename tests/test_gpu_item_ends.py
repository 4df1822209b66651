"""The end of an item in the long-run kernel: both row warpgroups read the accumulators there, and the next item of the CTA
may overwrite them only when both have.  Few CTAs, each with many uncut items of one to a few K/V tiles, whose first P V is
close behind the end of the item before; gates, unaligned outputs and partials lengthen that end in different ways."""
import numpy as np
import pytest

import checks
import gpuharness as G
import workloads as W
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,head_dim", [((24, 4), 256), ((16, 2), 256), ((40, 8), 128)])
@pytest.mark.parametrize("max_ctas", [2, 5])
@pytest.mark.parametrize("entry", ["plain", "gated", "gated_off_16", "partial"])
def test_items_that_follow_one_another_keep_their_rows(heads, head_dim, max_ctas, entry):
    import torch
    runs = [40, 64, 70, 129, 45, 200]
    s = W.Session(W.Spec("ends", pkg.BF16, *heads, head_dim, 16, [0, 3, 64, 20, 150, 0], runs, seed=91), max_ctas=max_ctas)
    s.append()
    shift = 4 if entry == "gated_off_16" else 0   # elements between a 16-byte boundary and gates / out
    gates = torch.empty(s.q.numel() + shift, dtype=s.tdtype, device=s.device).normal_(0, 2)[shift:].view(s.q.shape)
    out = torch.zeros(s.q.numel() + shift, dtype=s.tdtype, device=s.device)[shift:].view(s.q.shape)
    o, m, l = (torch.zeros(x, device=s.device) for x in (s.q.shape, s.q.shape[:2], s.q.shape[:2]))

    def run():
        if entry == "partial":
            s.gqa.attend_partial(s.pages, s.table, 0, s.q, o, m, l)
        elif entry == "plain":
            s.gqa.attend(s.pages, s.table, 0, s.q, out)
        else:
            s.gqa.attend_gated(s.pages, s.table, 0, s.q, gates, out)
        s.ctx.sync()
        return o.cpu().numpy().copy() if entry == "partial" else checks.to_numpy_bits(out).reshape(s.q.shape).copy()

    first = run()
    stats = s.gqa.plan_stats()
    assert stats["chunk_ctas"] == max_ctas and stats["chunk_items"] >= 4 * max_ctas
    expected, rows = checks.oracle_attention(s)
    expected = expected.astype(np.float64)
    got = first.astype(np.float64) if entry == "partial" else O.decode(first, pkg.BF16).astype(np.float64)
    if entry.startswith("gated"):
        expected = expected / (1.0 + np.exp(-O.decode(checks.to_numpy_bits(gates), pkg.BF16).astype(np.float64)[rows]))
    diff = np.abs(got[rows] - expected)
    assert diff.max() <= 2e-2 and diff.mean() <= 2e-3, (diff.max(), diff.mean())
    for _ in range(20):
        assert np.array_equal(run(), first)
    assert s.gqa.device_status() == 0
    s.close()
