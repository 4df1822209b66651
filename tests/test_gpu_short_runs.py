"""Short query runs and rows at one position on the tcgen05 kernel: weights as precise as the decode kernel's, values that
are not finite kept from the rows that must not see them, buffers it cannot address refused before anything is launched."""
import numpy as np
import pytest

import checks
import gpuharness as G
import workloads as W
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


def _partial(s):
    import torch
    o, m, l = (torch.zeros(x, device=s.device) for x in (s.q.shape, s.q.shape[:2], s.q.shape[:2]))
    s.gqa.attend_partial(s.pages, s.table, 0, s.q, o, m, l)
    s.ctx.sync()
    return o


# the routes are those of split_runs: units enough, or long enough, for the long-run kernel
@pytest.mark.parametrize("dtype", [pkg.BF16, pkg.F16])
@pytest.mark.parametrize("heads,head_dim,contexts,run", [((40, 8), 128, [900] * 40, 8), ((16, 2), 256, [2500] * 24, 8), ((24, 4), 256, [9000] * 4, 8)])
@pytest.mark.parametrize("replay", [False, True])
def test_partials_of_short_runs_are_as_close_as_the_decode_kernel(dtype, heads, head_dim, contexts, run, replay):
    # One rounding of the weights to 16 bits, which is independent from key to key, leaves about 2^-8 / sqrt(3) * 0.72 of the
    # result in bf16 and an eighth of that in f16; the decode kernel comes to three quarters of it, two parts to 2^-16.
    s = W.Session(W.Spec("short", dtype, *heads, head_dim, 16, contexts, [run] * len(contexts), seed=51))
    if replay:
        s.gqa.reserve_replay()
        s.gqa.prepare(*s.spec.batch())
    assert s.gqa.plan_stats()["chunk_ctas"] > 0
    s.append()
    o = _partial(s)
    sample = list(range(0, len(contexts), 13))
    expected, rows = checks.oracle_attention(s, sample)
    got = o.cpu().numpy().astype(np.float64)[rows]
    error = np.linalg.norm(got - expected) / np.linalg.norm(expected)
    assert error <= {pkg.BF16: 1.2e-3, pkg.F16: 1.5e-4}[dtype] / 8, error
    s.close()


def _rows_of(s, request):
    cu = np.concatenate([[0], np.cumsum(s.spec.q_len)])
    return np.arange(cu[request], cu[request + 1])
