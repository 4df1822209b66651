"""The ring-fed f32 kernel: row counts around 4, 8 and 16, head sizes around its lane split, ragged ranges and pages that
are no power of two, cut units, gates and external partials."""
import numpy as np
import pytest

import checks
import workloads as W
import gpuharness as G
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,runs", [((3, 1), [1, 1, 1, 1]), ((8, 2), [1, 2, 1, 3]), ((5, 1), [1, 1, 3, 2]), ((16, 2), [1, 2, 1, 5]),
                                        ((17, 1), [1, 1, 1, 1])])
@pytest.mark.parametrize("head_dim,page", [(32, 1), (96, 12), (128, 16), (160, 7), (256, 16)])
def test_f32_decode_matches_the_oracle(heads, runs, head_dim, page):
    spec = W.Spec("f32-rows", pkg.F32, *heads, head_dim, page, [1, 7, 1037, 2600], runs, seed=5)
    s = W.Session(spec)
    s.append()
    s.attend()
    s.ctx.sync()
    checks.assert_attention_close(s)
    s.close()


@pytest.mark.parametrize("head_dim", [128, 256])
def test_f32_gates_and_partials(head_dim):
    import torch
    spec = W.Spec("f32-rows", pkg.F32, 8, 2, head_dim, 16, [40, 9000], [1, 1], seed=6)
    s = W.Session(spec)
    s.append()
    gates = 2 * torch.randn_like(s.q)
    s.gqa.attend_gated(s.pages, s.table, 0, s.q, gates, s.out)
    o, m, l = torch.zeros_like(s.q), torch.zeros(s.q.shape[:2], device=s.device), torch.zeros(s.q.shape[:2], device=s.device)
    s.gqa.attend_partial(s.pages, s.table, 0, s.q, o, m, l)
    s.ctx.sync()
    expected, rows = checks.oracle_attention(s)
    got = checks.to_numpy_bits(o)[rows]
    assert np.abs(got - expected).max() <= 2e-5
    g = checks.to_numpy_bits(gates).astype(np.float64)[rows]
    assert np.abs(checks.to_numpy_bits(s.out)[rows] - expected / (1.0 + np.exp(-g))).max() <= 2e-5
    assert torch.isfinite(m).all() and (l >= 1.0).all()
    s.close()
