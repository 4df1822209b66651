"""The tensor-core kernel of the odd 16-bit profiles where its split weights could show: a dominant key over a long flat tail
in f16, infinities in V, buffers on 2-byte boundaries; the f32 kernel against the staged one; the static entry point."""
import numpy as np
import pytest

import checks
import workloads as W
import gpuharness as G
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


def _partial(s):
    import torch
    out = [torch.zeros(x, device=s.device) for x in (s.q.shape, s.q.shape[:2], s.q.shape[:2])]
    s.gqa.attend_partial(s.pages, s.table, 0, s.q, *out)
    s.ctx.sync()
    return [x.cpu().numpy().astype(np.float64) for x in out]


@pytest.mark.parametrize("dtype", [pkg.F16, pkg.BF16])
@pytest.mark.parametrize("head_dim", [96, 200])
@pytest.mark.parametrize("below", [17.5, 21.0, 26.0])   # log2 of the dominant key's weight over a tail key's
def test_a_long_tail_under_a_dominant_key_keeps_its_weights(dtype, head_dim, below):
    # Scores are set through one element of q and K: the tail's all are 0, one key's is `below` in log2.  V is 0 for that key
    # and about 1 for the tail, so that the partial is the tail's share, n 2^-below of the whole.
    import torch
    n = 6000
    answers = {}
    for mode in (pkg.KERNEL_AUTO, pkg.KERNEL_GENERIC):
        s = W.Session(W.Spec("tail", dtype, 4, 2, head_dim, 12, [n], [1], seed=71), kernel_mode=mode)
        pages = s.arena.view(s.arena.shape[0], 2, 2, 12, head_dim)
        ids = s.spec.block_tables[0]
        pages[:, 0] = 0
        pages[:, 1] = (1.0 + 0.25 * torch.randn(pages[:, 1].shape, generator=torch.Generator("cuda").manual_seed(3), device="cuda")).to(s.tdtype)
        s.q.zero_()
        s.q[..., 0] = 8.0
        key = 64  # in the first warp's share of the first item
        pages[int(ids[key // 12]), 0, :, key % 12, 0] = below * np.log(2.0) / (8.0 * s.spec.scale)
        pages[int(ids[key // 12]), 1, :, key % 12] = 0
        o, m, l = _partial(s)
        expected, rows = checks.oracle_attention(s)
        answers[mode] = np.linalg.norm(o[rows] - expected) / np.linalg.norm(expected)
        score = float(pages[int(ids[key // 12]), 0, 0, key % 12, 0]) * 8.0 * s.spec.scale
        assert np.allclose(m, score, rtol=1e-6) and np.allclose(l, 1.0 + n * np.exp(-score), rtol=1e-5)
        s.close()
    assert answers[pkg.KERNEL_AUTO] <= max(2e-6, 2 * answers[pkg.KERNEL_GENERIC]), answers


@pytest.mark.parametrize("dtype", [pkg.F16, pkg.BF16])
@pytest.mark.parametrize("entry", ["partial", "gated"])
def test_infinities_stay_infinities(dtype, entry):
    import torch
    s = W.Session(W.Spec("inf", dtype, 12, 4, 96, 12, [5000, 30], [1, 2], seed=72))
    s.append()
    gates = torch.randn(s.q.shape, generator=torch.Generator("cuda").manual_seed(5), device="cuda").to(s.tdtype)

    def run():
        if entry == "partial":
            return _partial(s)[0]
        s.gqa.attend_gated(s.pages, s.table, 0, s.q, gates, s.out)
        s.ctx.sync()
        return s.out.float().cpu().numpy()

    clean = run()
    pages = s.arena.view(s.arena.shape[0], 2, 4, 12, 96)
    expected = clean.copy()
    for request, position, head, column, value in ((0, 700, 0, 1, np.inf), (0, 4100, 1, 95, -np.inf), (0, 33, 2, 40, np.nan), (1, 4, 3, 7, np.inf),
                                                   (0, 100, 3, 0, np.inf), (0, 3000, 3, 0, -np.inf)):
        pages[int(s.spec.block_tables[request][position // 12]), 1, head, position % 12, column] = value
        rows = slice(0, 1) if request == 0 else slice(1, 3)
        at = expected[rows, 3 * head:3 * head + 3, column]
        expected[rows, 3 * head:3 * head + 3, column] = np.nan if np.isinf(at).all() else value   # Inf - Inf
    dirty = run()
    assert np.array_equal(dirty, expected, equal_nan=True)
    s.close()


@pytest.mark.parametrize("dtype", [pkg.F16, pkg.BF16])
@pytest.mark.parametrize("head_dim,page", [(96, 12), (200, 8), (8, 16)])
@pytest.mark.parametrize("where", ["q", "out", "arena", "gated"])
def test_buffers_on_two_byte_boundaries_give_the_same_bits(dtype, head_dim, page, where):
    import torch
    s = W.Session(W.Spec("shift", dtype, 6, 2, head_dim, page, [500, 70, 2300], [1, 2, 9], seed=73))
    s.append()

    def shifted(x):
        y = torch.zeros(x.numel() + 1, dtype=s.tdtype, device=s.device)[1:].view(x.shape)
        y.copy_(x)
        return y

    q, out, pages = s.q, torch.zeros_like(s.q), s.pages
    gates = torch.randn(s.q.shape, device="cuda").to(s.tdtype) if where == "gated" else None
    call = (lambda p, a, b: s.gqa.attend_gated(p, s.table, 0, a, gates, b)) if gates is not None else (lambda p, a, b: s.gqa.attend(p, s.table, 0, a, b))
    call(pages, q, out)
    s.ctx.sync()
    wanted = checks.to_numpy_bits(out).copy()
    held = None
    if where in ("q", "gated"):
        q = shifted(s.q)
    if where in ("out", "gated"):
        out = shifted(torch.zeros_like(out))
    if where == "arena":
        held = shifted(s.arena)
        pages = pkg.PageArena(s.ctx, s.spec.num_pages, s.spec.page_bytes, device_ptr=held)
    torch.cuda.synchronize()
    call(pages, q, out)
    s.ctx.sync()
    assert np.array_equal(checks.to_numpy_bits(out), wanted)
    if held is not None:
        pages.close()
    s.close()


@pytest.mark.parametrize("heads,head_dim", [((8, 2), 128), ((16, 2), 256), ((3, 1), 32)])
def test_f32_kernels_agree_on_partials(heads, head_dim):
    import torch
    found = []
    for mode in (pkg.KERNEL_AUTO, pkg.KERNEL_GENERIC):
        s = W.Session(W.Spec("f32", pkg.F32, *heads, head_dim, 16, [4000, 33, 900], [1, 3, 2], seed=74), kernel_mode=mode)
        s.append()
        found.append(_partial(s))
        s.close()
    # other sums in another order, and so other last bits: two kernels and not one
    assert not np.array_equal(found[0][0], found[1][0])
    for a, b in zip(*found):
        assert np.abs(a - b).max() <= 2e-5 * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("dtype,heads,head_dim,page,mode", [(pkg.BF16, (24, 8), 96, 12, pkg.KERNEL_AUTO), (pkg.F16, (16, 2), 200, 8, pkg.KERNEL_AUTO),
                                                            (pkg.F32, (8, 2), 128, 16, pkg.KERNEL_AUTO), (pkg.BF16, (24, 8), 96, 12, pkg.KERNEL_GENERIC),
                                                            (pkg.F32, (8, 2), 128, 16, pkg.KERNEL_GENERIC)])
def test_the_static_entry_point_takes_the_same_kernel(dtype, heads, head_dim, page, mode):
    # the same plan, kernel and reduce pass: the same bits (the static scratch holds plans of up to PSI_STATIC_MAX_CTAS)
    import torch
    s = W.Session(W.Spec("static", dtype, *heads, head_dim, page, [2600, 70, 900], [1, 2, 1], seed=75), kernel_mode=mode, max_ctas=64)
    s.append()
    s.attend()
    out = torch.zeros_like(s.out)
    config = pkg.GQAConfig(*heads, head_dim, s.spec.scale, s.spec.page_bytes, dtype, s.layout, s.spec.num_tokens, pkg.PLAN_BALANCED, mode, 64)
    pkg.attend_static(0, s.stream.cuda_stream, config, s.arena, s.table.page_ids_buffer(), *s.spec.batch(), s.spec.layer, s.q, out)
    s.ctx.sync()
    torch.cuda.synchronize()
    assert np.array_equal(checks.to_numpy_bits(out), checks.to_numpy_bits(s.out))
    s.close()
