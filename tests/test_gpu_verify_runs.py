"""Short query runs (verification of a draft): which kernel takes them, and the same numbers from either."""
import numpy as np
import pytest

import checks
import workloads as W
import gpuharness as G

pkg = G.pkg
pytestmark = pytest.mark.gpu

# (heads, head_dim, contexts, runs, long-run kernel expected): two tiles and more go there once reading the K/V once instead
# of once per tile saves more than cutting the units costs
CASES = [((40, 8), 128, [300], [4], False), ((40, 8), 128, [5000], [4], False), ((16, 2), 256, [3000] * 5, [3] * 5, False),
         ((16, 2), 256, [3000] * 4, [3] * 4, False), ((24, 4), 256, [700, 9000, 64, 4000], [8, 9, 2, 43], True),
         ((24, 4), 256, [9000] * 8, [2] * 8, False), ((18, 2), 128, [900, 40], [2, 1], False), ((12, 2), 128, [4000], [11], True),
         ((40, 8), 128, [900] * 40, [4] * 40, True), ((16, 2), 256, [2500] * 24, [8, 3] * 12, True), ((24, 4), 256, [9000] * 8, [3] * 8, True)]


@pytest.mark.parametrize("heads,head_dim,contexts,runs,long_run", CASES)
@pytest.mark.parametrize("replay", [False, True])
def test_short_runs_match_the_oracle_on_either_kernel(heads, head_dim, contexts, runs, long_run, replay):
    spec = W.Spec("verify", pkg.BF16, *heads, head_dim, 16, contexts, runs, seed=41)
    s = W.Session(spec)
    if replay:
        s.gqa.reserve_replay()
        s.gqa.prepare(*spec.batch())
    assert (s.gqa.plan_stats()["chunk_ctas"] > 0) == long_run
    s.append()
    s.attend()
    s.ctx.sync()
    checks.assert_attention_close(s)
    s.gqa.append_attend(s.pages, s.table, 0, s.k, s.v, s.q, s.out)
    s.ctx.sync()
    checks.assert_attention_close(s)
    assert s.gqa.device_status() == 0
    s.close()
