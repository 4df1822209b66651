"""A page table that the caller's own kernels fill through its device address, in the order of the context's stream."""
import numpy as np
import pytest

import checks
import workloads as W
import gpuharness as G
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


def _table_tensor(s):
    import torch

    class Address:
        def __init__(self, pointer, shape):
            self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i4", "data": (pointer, False), "version": 3}

    layout = s.layout
    shape = (layout.num_req_slots, layout.num_gqa_layers, layout.num_blocks * layout.num_page_ids_per_block)
    return torch.as_tensor(Address(int(s.table.page_ids_buffer()), shape), device=s.device)


@pytest.mark.parametrize("dtype,heads,head_dim,page", [(pkg.BF16, (40, 8), 128, 8), (pkg.BF16, (16, 2), 256, 16), (pkg.F16, (16, 4), 64, 16),
                                                       (pkg.F32, (8, 2), 128, 16), (pkg.BF16, (24, 8), 96, 12)])
@pytest.mark.parametrize("runs", [[1] * 6, [8] * 6, [200] + [1] * 5])
def test_a_table_filled_by_a_kernel_directly_before_the_launch(dtype, heads, head_dim, page, runs):
    import torch
    spec = W.Spec("table", dtype, *heads, head_dim, page, [2000, 65, 900, 16, 3000, 700], runs, seed=61)
    s = W.Session(spec)
    s.append()
    s.attend()
    s.ctx.sync()
    checks.assert_attention_close(s)
    table = _table_tensor(s)
    right = table.clone()
    wrong = right.flip(2).contiguous()
    rng = np.random.default_rng(head_dim)
    s.gqa.set_norm_rope(pkg.NormRopeConfig(head_dim, 1e-6, 1e6, 0, 1, 1, 1, 1, 1, 0),
                        *[O.encode(1.0 + 0.1 * rng.standard_normal(head_dim).astype(np.float32), O.BF16).tolist() for _ in range(2)])
    q_in, q_out = s.q.clone(), torch.zeros_like(s.q)
    # the front stage writes k and v through the right table whatever the table held before
    before = s.arena.clone()
    s.gqa.norm_rope_append(s.pages, s.table, 0, q_in, s.k, s.v, q_out)
    s.ctx.sync()
    wanted, wanted_q = s.arena.clone(), q_out.clone()
    assert not torch.equal(before, wanted)
    for step in range(20):
        s.arena.copy_(before)
        table.copy_(wrong)
        torch.add(right, 0, out=table)
        s.gqa.norm_rope_append(s.pages, s.table, 0, q_in, s.k, s.v, q_out)
        table.copy_(wrong)
        s.ctx.sync()
        assert torch.equal(s.arena.view(torch.uint8), wanted.view(torch.uint8)) and torch.equal(q_out, wanted_q), step
    s.arena.copy_(before)
    for step in range(20):
        s.out.zero_()
        table.copy_(wrong)
        torch.add(right, 0, out=table)
        s.attend()
        table.copy_(wrong)
        torch.cuda.synchronize()
        checks.assert_attention_close(s, [step % 6])
    s.close()
