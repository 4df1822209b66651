"""Long query runs whose group is no divisor of 128: an item's rows are packed (token, head) pairs, so tokens straddle
the 16-row tiles; and the epilogue's gates and outputs at the 8-byte alignment the entry point asks for."""
import numpy as np
import pytest

import checks
import gpuharness as G
import workloads as W
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [pkg.KERNEL_AUTO, pkg.KERNEL_MMA_SYNC])
@pytest.mark.parametrize("heads,head_dim", [((24, 4), 256), ((14, 2), 128), ((10, 2), 128), ((34, 2), 128)])
@pytest.mark.parametrize("shift", [0, 4])  # elements between a 16-byte boundary and gates / out
def test_packed_rows_and_gates_of_long_runs(heads, head_dim, engine, shift):
    import torch
    per_item = 128 // min(16, heads[0] // heads[1])
    runs = [1, 5 * per_item + 1, per_item - 1, 2 * per_item, 300]
    spec = W.Spec("packed", pkg.BF16, heads[0], heads[1], head_dim, 16, [70, 0, 333, 16, 2500], runs, seed=31)
    s = W.Session(spec, kernel_mode=engine)
    s.append()
    gates = torch.empty(s.q.numel() + shift, dtype=s.tdtype, device=s.device).normal_(0, 2)[shift:].view(s.q.shape)
    out = torch.zeros(s.q.numel() + shift, dtype=s.tdtype, device=s.device)[shift:].view(s.q.shape)
    s.gqa.attend_gated(s.pages, s.table, 0, s.q, gates, out)
    s.ctx.sync()
    attention, rows = checks.oracle_attention(s)
    g = O.decode(checks.to_numpy_bits(gates), spec.dtype).astype(np.float64)[rows]
    diff = np.abs(O.decode(checks.to_numpy_bits(out), spec.dtype)[rows] - attention.astype(np.float64) / (1.0 + np.exp(-g)))
    assert diff.max() <= 2e-2 and diff.mean() <= 2e-3, (diff.max(), diff.mean())
    assert s.gqa.device_status() == 0
    s.close()
