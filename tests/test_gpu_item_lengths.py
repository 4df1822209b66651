"""Steps on both sides of the lines where a kernel takes more warps for long items, with units cut between CTAs (merged in the
launch), and long runs whose items hold one K/V tile and more, so that the two streams of head_dim 128 end on either side."""
import numpy as np
import pytest

import checks
import gpuharness as G
import workloads as W
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,heads,head_dim,page,line", [
    (pkg.F16, (16, 4), 64, 16, 32), (pkg.BF16, (32, 8), 64, 8, 32),                              # attend_mma
    (pkg.BF16, (24, 8), 96, 12, 64), (pkg.F16, (12, 4), 48, 16, 64), (pkg.BF16, (6, 2), 56, 7, 64),   # attend_mma_any
    (pkg.F32, (32, 8), 128, 16, 20), (pkg.F32, (8, 2), 64, 12, 20)])                                   # attend_f32
@pytest.mark.parametrize("length", ["short", "long", "one"])
def test_steps_on_both_sides_of_the_line(dtype, heads, head_dim, page, line, length):
    contexts = {"short": [0, 1, 15, 16, 17, 40, 130, 257, 300, 33], "long": [3000, 2900, 1, 3100, 3300, 2048, 3007, 2999], "one": [2500]}[length]
    contexts = contexts * (6 if length == "long" and line == 64 else 2 if length != "one" else 1)
    spec = W.Spec("length", dtype, *heads, head_dim, page, contexts, [1 + i % 2 for i in range(len(contexts))], seed=81)
    s = W.Session(spec)
    s.append()
    s.attend()
    s.ctx.sync()
    stats = s.gqa.plan_stats()
    per_item = stats["kv_tiles"] // stats["items"]
    assert length == "one" or (per_item >= line) == (length == "long"), per_item
    checks.assert_attention_close(s)
    first = checks.to_numpy_bits(s.out).copy()
    for _ in range(2):  # the arrival counters are back at zero, and pieces meet in the plan's order whoever is last
        s.out.zero_()
        s.attend()
        s.ctx.sync()
        assert np.array_equal(checks.to_numpy_bits(s.out), first)
    s.close()


@pytest.mark.parametrize("heads,head_dim", [((40, 8), 128), ((24, 4), 256)])
@pytest.mark.parametrize("page", [8, 16, 64])
@pytest.mark.parametrize("max_ctas", [0, 3])
def test_long_runs_of_few_tiles(heads, head_dim, page, max_ctas):
    contexts, run = [0, 24, 25, 64, 100, 128, 190, 256, 300, 448], 40
    spec = W.Spec("tiles", pkg.BF16, *heads, head_dim, page, contexts, [run] * len(contexts), seed=82)
    s = W.Session(spec, max_ctas=max_ctas)
    s.append()
    s.attend()
    s.ctx.sync()
    assert s.gqa.plan_stats()["chunk_tcgen05_launches"] == 1
    checks.assert_attention_close(s)
    assert s.gqa.device_status() == 0
    s.close()


@pytest.mark.parametrize("heads,head_dim", [((40, 8), 128), ((24, 4), 256)])
def test_a_gate_that_is_no_number_stays_alone(heads, head_dim):
    import torch
    s = W.Session(W.Spec("gates", pkg.BF16, *heads, head_dim, 16, [70, 0], [50, 33], seed=83))
    s.append()
    gates = (4 * torch.randn(s.q.shape, generator=torch.Generator("cuda").manual_seed(7), device="cuda")).to(s.tdtype)
    gates[3, 1, 5], gates[40, 0, 7], gates[60, 2, 64] = float("inf"), -float("inf"), 200.0

    def run():
        s.gqa.attend_gated(s.pages, s.table, 0, s.q, gates, s.out)
        s.ctx.sync()
        return s.out.float().cpu().numpy()

    expected = run()
    attention, rows = checks.oracle_attention(s)
    g = O.decode(checks.to_numpy_bits(gates), pkg.BF16).astype(np.float64)[rows]
    diff = np.abs(expected[rows] - attention.astype(np.float64) / (1.0 + np.exp(-g)))
    assert diff.max() <= 2e-2 and diff.mean() <= 2e-3
    for token, head, column in ((0, 0, 0), (17, 2, 33), (49, 3, head_dim - 1), (82, 1, 66)):
        gates[token, head, column] = float("nan")
        expected[token, head, column] = np.nan
    assert np.array_equal(run(), expected, equal_nan=True)
    s.close()
