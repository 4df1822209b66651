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


@pytest.mark.parametrize("dtype", [pkg.BF16, pkg.F16])
@pytest.mark.parametrize("heads,head_dim,context,count", [((40, 8), 128, 897, 40), ((16, 2), 256, 2500, 24), ((24, 4), 256, 8130, 4)])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_a_value_that_is_not_finite_stays_in_the_rows_that_see_it(dtype, heads, head_dim, context, count, bad):
    import torch
    run, hit = 8, 5   # value column 3 of KV head 1 of the sixth token of request 1; column 70 of a key of its history
    s = W.Session(W.Spec("inf", dtype, *heads, head_dim, 16, [context] * count, [run] * count, seed=52))
    s.append()
    assert s.gqa.plan_stats()["chunk_ctas"] > 0
    clean = _partial(s).cpu().numpy()
    rows, group = _rows_of(s, 1), heads[0] // heads[1]
    pages = s.arena.view(s.arena.shape[0], 2, heads[1], 16, head_dim)
    for position, column in ((context + hit, 3), (context // 2, 60)):
        page = int(s.spec.block_tables[1][position // 16])
        pages[page, 1, 1, position % 16, column] = bad
    dirty = _partial(s).cpu().numpy()
    expected = clean.copy()
    expected[rows[hit:], group:2 * group, 3] = bad
    expected[rows, group:2 * group, 60] = bad
    same = np.isfinite(expected)
    assert np.array_equal(np.isfinite(dirty), same)
    assert np.array_equal(dirty[same], clean[same])
    assert np.array_equal(dirty[~same], expected[~same], equal_nan=True)
    assert s.gqa.device_status() == 0
    s.close()


@pytest.mark.parametrize("engine", [pkg.KERNEL_AUTO, pkg.KERNEL_MMA_SYNC, pkg.KERNEL_MMA_TMA])
@pytest.mark.parametrize("runs,contexts", [([1] * 3, [70, 9, 300]), ([8] * 40, [900] * 40), ([300, 1], [20, 400])])
def test_unaligned_buffers_are_refused_before_anything_is_launched(engine, runs, contexts):
    # host side only: no kernel sees one of these pointers
    import torch
    s = W.Session(W.Spec("shift", pkg.BF16, 40, 8, 128, 16, contexts, runs, seed=53), kernel_mode=engine)
    s.append()
    s.attend()
    s.ctx.sync()
    good = checks.to_numpy_bits(s.out).copy()

    def shifted(elements):
        x = torch.zeros(s.q.numel() + elements, dtype=s.tdtype, device=s.device)[elements:].view(s.q.shape)
        x.copy_(s.q)
        return x

    o, m, l = (torch.zeros(x, device=s.device) for x in (s.q.shape, s.q.shape[:2], s.q.shape[:2]))
    torch.cuda.synchronize()
    for q, out in ((shifted(4), s.out), (shifted(1), s.out), (s.q, shifted(2))):
        before = s.ctx.launch_count
        with pytest.raises(pkg.PsiError, match="cudaErrorMisalignedAddress"):
            s.gqa.attend(s.pages, s.table, 0, q, out)
        with pytest.raises(pkg.PsiError, match="cudaErrorMisalignedAddress"):
            s.gqa.append_attend(s.pages, s.table, 0, s.k, s.v, q, out)
        if q is not s.q:
            with pytest.raises(pkg.PsiError, match="cudaErrorMisalignedAddress"):
                s.gqa.attend_partial(s.pages, s.table, 0, q, o, m, l)
        assert s.ctx.launch_count == before
    off = pkg.PageArena(s.ctx, s.spec.num_pages - 1, s.spec.page_bytes, device_ptr=s.arena.view(-1)[4:])
    with pytest.raises(pkg.PsiError, match="cudaErrorMisalignedAddress"):
        s.gqa.attend(off, s.table, 0, s.q, s.out)
    off.close()
    s.out.zero_()
    s.attend()
    s.ctx.sync()
    assert np.array_equal(checks.to_numpy_bits(s.out), good)
    s.close()


# (first: the decode kernel in place beats the long-run kernel behind a pull of 6 MiB; second: the pull of 1.2 MiB is worth it)
@pytest.mark.parametrize("heads,head_dim,contexts,long_run", [((32, 8), 128, [1500 + 23 * i for i in range(64)], False),
                                                               ((16, 2), 256, [512 + 1050 * i for i in range(16)], True)])
def test_host_steps_with_short_runs_take_the_long_run_kernel_where_it_saves_the_pull(heads, head_dim, contexts, long_run):
    import torch
    s = W.Session(W.Spec("host", pkg.BF16, *heads, head_dim, 16, contexts, [8] * len(contexts), seed=54))
    assert s.gqa.plan_stats()["chunk_ctas"] > 0
    host = [x.cpu().pin_memory() for x in (s.k, s.v, s.q)]
    out = torch.zeros_like(host[2]).pin_memory()
    before = checks.to_numpy_bits(s.arena)
    s.gqa.step_host(s.pages, s.table, 0, *s.spec.batch(), *host, out)
    assert (s.gqa.plan_stats()["chunk_ctas"] > 0) == long_run
    assert np.array_equal(checks.to_numpy_bits(s.arena).reshape(-1), checks.expected_arena_after_append(s, before))
    s.out.copy_(out.cuda())
    checks.assert_attention_close(s)
    s.close()
