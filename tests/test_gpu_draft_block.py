"""A drafter's step: block rows that all stand at the last history position share one pass over the history; the block's own
attention and the merge of the two."""
import numpy as np
import pytest

import gpuharness as G
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


def _rig(dtype, heads, head_dim, page, contexts, max_tokens, seed=3):
    rng = np.random.default_rng(seed)
    counts = [-(-(c + 1) // page) for c in contexts]
    rig = G.Rig(dtype, *heads, head_dim, page, head_dim ** -0.5, (len(contexts), 1, max(counts), 1), max_tokens,
                arena_f32=rng.standard_normal((sum(counts), 2 * heads[1] * page * head_dim)).astype(np.float32))
    ids = rng.permutation(sum(counts))
    for slot, n in enumerate(counts):
        rig.set_pages(slot, 0, ids[:n])
        ids = ids[n:]
    return rig


@pytest.mark.parametrize("dtype,heads,head_dim,page", [(pkg.BF16, (40, 8), 128, 8), (pkg.BF16, (16, 2), 256, 16), (pkg.F16, (16, 4), 64, 16),
                                                       (pkg.F32, (8, 2), 128, 16), (pkg.BF16, (24, 8), 96, 12), (pkg.F32, (6, 2), 40, 16)])
@pytest.mark.parametrize("blocks", [[7, 7, 7], [1, 2, 1, 30], [3]])
@pytest.mark.parametrize("replay", [False, True])
def test_rows_at_one_position_match_the_oracle(dtype, heads, head_dim, page, blocks, replay):
    import torch
    contexts = [2600, 65, 900, 16][:len(blocks)]
    t = sum(blocks)
    rig = _rig(dtype, heads, head_dim, page, contexts, t)
    slots = np.repeat(np.arange(len(blocks)), blocks)
    positions = np.repeat(contexts, blocks) - 1
    if replay:
        rig.gqa.reserve_replay()
    rig.gqa.prepare(slots.tolist(), positions.tolist(), list(range(t + 1)))
    q = G.to_device(np.random.default_rng(4).standard_normal((t, heads[0], head_dim)).astype(np.float32), dtype).view(t, heads[0], head_dim)
    o, m, l = (torch.zeros(s, device="cuda") for s in ((t, heads[0], head_dim), (t, heads[0]), (t, heads[0])))
    out = torch.zeros_like(q)
    rig.gqa.attend_partial(rig.pages, rig.table, 0, q, o, m, l)
    rig.gqa.attend(rig.pages, rig.table, 0, q, out)
    rig.ctx.sync()
    expected = rig.oracle_attention(q, slots.tolist(), positions.tolist())
    tol = 2e-5 if dtype == pkg.F32 else 2e-2
    assert np.abs(o.cpu().numpy().reshape(expected.shape) - expected).max() <= tol
    assert np.abs(O.decode(G.bits_of(out), dtype).reshape(expected.shape) - expected).max() <= tol
    assert rig.gqa.device_status() == 0
    rig.close()


@pytest.mark.parametrize("dtype", [pkg.BF16, pkg.F32])
def test_fused_rows_at_one_position_see_their_own_key(dtype):
    # append_attend: every request of the batch sees the history and the K/V row it brings itself, also where two of them
    # stand at one position of one slot; f32 appends first, so there the last writer's row is what all of them read, and
    # all bring the same
    import torch
    heads, d, contexts = (8, 2), 128, [700, 33]
    rig = _rig(dtype, heads, d, 16, contexts, 6)
    slots, positions = [0, 0, 0, 1, 1, 1], [700, 700, 700, 33, 33, 33]
    rng = np.random.default_rng(5)
    q, k, v = (G.to_device(rng.standard_normal((6, h, d)).astype(np.float32), dtype).view(6, h, d) for h in (heads[0], heads[1], heads[1]))
    if dtype == pkg.F32:
        for x in (k, v):
            x[1:3], x[4:6] = x[0], x[3]
    out, one = torch.zeros_like(q), torch.zeros_like(q)
    rig.gqa.prepare(slots, positions, list(range(7)))
    rig.gqa.append_attend(rig.pages, rig.table, 0, k, v, q, out)
    for i in range(6):
        rig.gqa.prepare([slots[i]], [positions[i]], [0, 1])
        rig.gqa.append_attend(rig.pages, rig.table, 0, k[i], v[i], q[i], one[i])
    rig.ctx.sync()
    tol = 2e-5 if dtype == pkg.F32 else 2e-2
    assert np.abs(O.decode(G.bits_of(out), dtype) - O.decode(G.bits_of(one), dtype)).max() <= tol
    rig.close()


@pytest.mark.parametrize("dtype,heads,head_dim", [(pkg.BF16, (5, 1), 64), (pkg.BF16, (40, 8), 128), (pkg.F16, (6, 2), 256), (pkg.F32, (4, 2), 128)])
@pytest.mark.parametrize("block", [1, 7, 8, 9, 40, 256])
@pytest.mark.parametrize("partials", [2, 3, 5])
def test_block_partial_and_combine_match_the_oracle(dtype, heads, head_dim, block, partials):
    import torch
    t, (hq, hkv) = 2 * block, heads
    rng = np.random.default_rng(block + head_dim)
    rig = _rig(dtype, heads, head_dim, 16, [16], t)
    bits = [O.encode(rng.standard_normal((t, h, head_dim)).astype(np.float32), dtype) for h in (hq, hkv, hkv)]
    q, k, v = (G.bits_to_device(b, dtype) for b in bits)
    found = []
    for i in range(partials):
        o, m, l = (torch.zeros(s, device="cuda") for s in ((t, hq, head_dim), (t, hq), (t, hq)))
        if i < partials - 1:
            rig.gqa.block_partial(q, k, v, t, block, o, m, l)
            if i == 0:
                first = (o, m, l)
            elif i == 1:
                o.mul_(-2.0), m.add_(1.0)  # another partial of the same rows
        else:
            m.fill_(-float("inf"))  # one that saw no key
        found.append((o, m, l))
    out = torch.zeros((t, hq, head_dim), dtype=G.torch_dtype(dtype), device="cuda")
    rig.gqa.combine(*zip(*found), t, out)
    rig.ctx.sync()
    want = O.block_sdpa(*(b.reshape(-1) for b in bits), dtype, t, block, hq, hkv, head_dim, rig.scale)
    for got, expected in zip(first, want):
        got, expected = got.cpu().numpy().reshape(-1), np.asarray(expected, dtype=np.float64).reshape(-1)
        assert np.abs(got - expected).max() <= 2e-5 * max(1.0, np.abs(expected).max())
    o, m, l = (np.stack([x[i].cpu().numpy().astype(np.float64) for x in found]) for i in range(3))
    w = np.exp(m - m.max(0)) * l
    merged = (w[..., None] * o).sum(0) / w.sum(0)[..., None]
    ulp = {pkg.F32: 2.0 ** -20, pkg.BF16: 2.0 ** -8, pkg.F16: 2.0 ** -11}[dtype]
    assert np.abs(O.decode(G.bits_of(out), dtype).reshape(merged.shape) - merged).max() <= 1.01 * ulp * max(1.0, np.abs(merged).max())
    rig.close()
