"""Cut units of the f32 and the odd-profile kernel on both sides of the line between the merge in the launch and the reduce
launch: two pieces to as many as the device has CTAs, several steps in one, also as a replay reservation launches them."""
import numpy as np
import pytest

import checks
import gpuharness as G
import workloads as W

pkg = G.pkg
pytestmark = pytest.mark.gpu


def _partial(s):
    import torch
    o, m, l = (torch.zeros(x, device=s.device) for x in (s.q.shape, s.q.shape[:2], s.q.shape[:2]))
    s.gqa.attend_partial(s.pages, s.table, 0, s.q, o, m, l)
    s.ctx.sync()
    return o, m.cpu().numpy(), l.cpu().numpy()


@pytest.mark.parametrize("dtype,heads,head_dim", [(pkg.F32, (16, 1), 128), (pkg.F32, (8, 2), 256), (pkg.F32, (16, 4), 64), (pkg.F32, (3, 1), 32),
                                                  (pkg.BF16, (16, 1), 160), (pkg.F16, (12, 2), 200), (pkg.BF16, (24, 8), 96)])
@pytest.mark.parametrize("contexts", [[5000], [2500, 3, 700], [300] * 12, [4000, 4000, 16, 1000]])
@pytest.mark.parametrize("replay", [False, True])
def test_units_of_few_and_of_many_pieces(dtype, heads, head_dim, contexts, replay):
    s = W.Session(W.Spec("merge", dtype, *heads, head_dim, 16, contexts, [1 + i % 2 for i in range(len(contexts))], seed=96))
    if replay:
        s.gqa.reserve_replay()
        s.gqa.prepare(*s.spec.batch())
    s.append()
    s.attend()
    s.ctx.sync()
    stats = s.gqa.plan_stats()
    assert stats["reduce_units"] > 0 or len(contexts) == 12
    checks.assert_attention_close(s)
    first = checks.to_numpy_bits(s.out).copy()
    for _ in range(2):  # the arrival counters are back at zero
        s.out.zero_()
        s.attend()
        s.ctx.sync()
        assert np.array_equal(checks.to_numpy_bits(s.out), first)
    assert s.gqa.device_status() == 0
    s.close()


@pytest.mark.parametrize("heads,head_dim,contexts", [((64, 8), 128, [700]), ((64, 8), 128, [2500]), ((8, 8), 64, [1500]), ((8, 1), 64, [5000])])
def test_an_infinite_maximum_weighs_nothing_in_a_cut_unit(heads, head_dim, contexts):
    # pieces whose maximum is not finite have no weight, the others none beside an infinite one: rows of zeros, l = 0, m = Inf
    # (pieces: one round trip of the merge, two of them, several threads a column, and the reduce launch)
    group = heads[0] // heads[1]
    for mode in (pkg.KERNEL_AUTO, pkg.KERNEL_GENERIC):
        s = W.Session(W.Spec("inf", pkg.F32, *heads, head_dim, 16, contexts, [1], seed=97), kernel_mode=mode)
        s.append()
        assert s.gqa.plan_stats()["reduce_units"] == heads[1]
        pages = s.arena.view(s.arena.shape[0], 2, heads[1], 16, head_dim)
        clean = [x if i else x.cpu().numpy() for i, x in enumerate(_partial(s))]
        hit = [0] if heads[1] == 1 else [2, 5]
        for head, position in zip(hit, (5, contexts[0] - 1)):   # in the first piece and in the last
            s.q[0, head * group:(head + 1) * group, 0] = 2.0
            pages[int(s.spec.block_tables[0][position // 16]), 0, head, position % 16, 0] = float("inf")
        o, m, l = _partial(s)
        o = o.cpu().numpy()
        rows = np.zeros(heads[0], dtype=bool)
        for head in hit:
            rows[head * group:(head + 1) * group] = True
        assert np.isposinf(m[0, rows]).all() and (l[0, rows] == 0.0).all() and (o[0, rows] == 0.0).all()
        for a, b in zip((o, m, l), clean):
            assert np.array_equal(a[0, ~rows], b[0, ~rows])
        s.close()
