"""Scores that are not finite on the long-run kernel: an infinity in K or in q is no number in the rows that see it, whatever
the head size, the number of streams and pieces, and the run's kind, as float64 has it; and an infinity in V stays in a row
however small its key's weight is."""
import numpy as np
import pytest

import gpuharness as G
import workloads as W

pkg = G.pkg
pytestmark = pytest.mark.gpu

PAGE = 16


def _float64(s, request, head):
    """(rows of the step, outputs, maxima) of one request and q head, from the bits the kernels see."""
    cu = np.concatenate([[0], np.cumsum(s.spec.q_len)])
    rows = np.arange(cu[request], cu[request + 1])
    first, kv_head = int(s.spec.context_lens[request]), head // (s.spec.num_q_heads // s.spec.num_kv_heads)
    pages = s.arena.view(s.arena.shape[0], 2, s.spec.num_kv_heads, PAGE, s.spec.head_dim)
    ids = np.asarray(s.spec.block_tables[request], dtype=np.int64)
    k, v = (pages[ids, which, kv_head].reshape(-1, s.spec.head_dim)[:first + len(rows)].double().cpu().numpy() for which in (0, 1))
    q = s.q[rows[0]:rows[-1] + 1, head].double().cpu().numpy()
    with np.errstate(all="ignore"):
        score = (q @ k.T) * s.spec.scale
        score[np.arange(len(k))[None] > first + np.arange(len(rows))[:, None]] = -np.inf
        top = score.max(axis=1)
        w = np.exp(score - top[:, None])
        return rows, (w @ v) / w.sum(axis=1, keepdims=True), top


def _run(s, entry, gates):
    import torch
    if entry == "partial":
        o, m, l = (torch.zeros(x, device=s.device) for x in (s.q.shape, s.q.shape[:2], s.q.shape[:2]))
        s.gqa.attend_partial(s.pages, s.table, 0, s.q, o, m, l)
        s.ctx.sync()
        return o.double().cpu().numpy(), m.cpu().numpy(), l.cpu().numpy()
    if entry == "gated":
        s.gqa.attend_gated(s.pages, s.table, 0, s.q, gates, s.out)
    else:
        s.gqa.attend(s.pages, s.table, 0, s.q, s.out)
    s.ctx.sync()
    return s.out.double().cpu().numpy(), None, None


# (profile, cached tokens, run, CTAs, whether units are cut); the short runs are those that take the fine weights
STEPS = {"whole-128": ((40, 8), 128, [300, 70], 40, 2, False), "whole-256": ((24, 4), 256, [300, 70], 40, 2, False),
         "cut-128": ((40, 8), 128, [6000, 70], 40, 0, True), "cut-256": ((24, 4), 256, [6000, 70], 40, 0, True),
         "short-128": ((40, 8), 128, [900] * 40, 8, 0, None), "short-256": ((16, 2), 256, [2500] * 24, 8, 0, None)}


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("where", ["k", "q"])
@pytest.mark.parametrize("entry", ["plain", "gated", "partial"])
def test_an_infinite_score_is_no_number(step, where, entry):
    import torch
    heads, head_dim, contexts, run, max_ctas, cut = STEPS[step]
    s = W.Session(W.Spec("inf", pkg.BF16, *heads, head_dim, PAGE, contexts, [run] * len(contexts), seed=61), max_ctas=max_ctas)
    s.append()
    stats, group = s.gqa.plan_stats(), heads[0] // heads[1]
    units = len(contexts) * heads[1] * -(-run // (128 // group))
    assert stats["chunk_ctas"] > 0 and (cut is None or (stats["chunk_items"] > units) == cut)
    gates = torch.randn(s.q.shape, generator=torch.Generator("cuda").manual_seed(5), device="cuda").to(s.tdtype)
    clean = _run(s, entry, gates)[0]
    head, context = group + 1, contexts[0]   # the second q head of KV head 1, request 0
    cu = int(s.spec.q_len[0])
    if where == "k":   # one key of the history, one of the step itself (seen by the rows from the 6th on); q decides the sign
        pages = s.arena.view(s.arena.shape[0], 2, heads[1], PAGE, head_dim)
        for position, column in ((context // 2 + 70, 3), (context + 5, 60)):
            pages[int(s.spec.block_tables[0][position // PAGE]), 0, 1, position % PAGE, column] = float("inf")
        touched = range(group, 2 * group)
    else:
        s.q[2, head, 7] = float("inf")
        touched = [head]
    out, m, l = _run(s, entry, gates)
    with np.errstate(all="ignore"):
        factor = 1.0 / (1.0 + np.exp(-gates.double().cpu().numpy())) if entry == "gated" else np.ones(s.q.shape)
    seen_nan = seen_number = 0
    for h in touched:
        rows, expected, top = _float64(s, 0, h)
        expected = expected * factor[rows, h]
        assert np.array_equal(np.isnan(out[rows, h]), np.isnan(expected)), h
        fine = np.isfinite(expected)
        assert np.abs(out[rows, h][fine] - expected[fine]).max(initial=0.0) <= 2e-2
        seen_nan += (~fine).any(axis=1).sum()
        seen_number += fine.all(axis=1).sum()
        if entry == "partial":
            assert np.array_equal(np.isposinf(m[rows, h]), np.isposinf(top)) and np.array_equal(np.isnan(l[rows, h]), np.isposinf(top))
    assert seen_nan > 0 and seen_number > 0
    others = np.ones(out.shape[:2], dtype=bool)
    others[:cu, list(touched)] = False
    assert np.array_equal(out[others], clean[others])
    assert s.gqa.device_status() == 0
    s.close()


@pytest.mark.parametrize("step", ["whole-128", "whole-256", "cut-128", "short-128"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_value_under_a_vanishing_weight_stays(step, bad):
    # request 0, KV head 1: one key outweighs all others by 2^300; V is not finite at a key of the next K/V tile
    heads, head_dim, contexts, run, max_ctas, _ = STEPS[step]
    s = W.Session(W.Spec("far", pkg.BF16, *heads, head_dim, PAGE, contexts, [run] * len(contexts), seed=62), max_ctas=max_ctas)
    s.append()
    assert s.gqa.plan_stats()["chunk_ctas"] > 0
    group, pages = heads[0] // heads[1], s.arena.view(s.arena.shape[0], 2, heads[1], PAGE, head_dim)

    def at(position):
        return int(s.spec.block_tables[0][position // PAGE]), position % PAGE

    rows = int(s.spec.q_len[0])
    s.q[:rows, group:2 * group, 0] = 16.0
    for page in s.spec.block_tables[0]:
        pages[int(page), 0, 1, :, 0] = 0.0
    page, row = at(10)
    pages[page, 0, 1, row, 0] = 300.0 * np.log(2.0) / (16.0 * s.spec.scale)
    page, row = at(100)
    pages[page, 1, 1, row, 9] = bad
    out = _run(s, "plain", None)[0][:rows, group:2 * group]
    assert not np.isfinite(out[..., 9]).any()
    assert np.isfinite(np.delete(out, 9, axis=2)).all()
    s.close()
