"""The static entry point plans as psi_gqa_prepare does, small steps in equal pieces among them: the same bits where both have as
many CTAs."""
import numpy as np
import pytest

import checks
import gpuharness as G
import workloads as W

pkg = G.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,heads,head_dim,page", [(pkg.BF16, (40, 8), 128, 8), (pkg.F16, (16, 4), 64, 16), (pkg.BF16, (16, 2), 256, 16), (pkg.BF16, (24, 8), 96, 12),
                                                       (pkg.BF16, (16, 2), 200, 8), (pkg.F32, (32, 8), 128, 16), (pkg.F32, (16, 2), 256, 16), (pkg.F32, (10, 2), 80, 16),
                                                       (pkg.BF16, (4, 2), 66, 16)])
@pytest.mark.parametrize("contexts", [[100], [777], [2500], [300] * 5, [40, 900, 3000]])
def test_small_steps_give_the_same_bits(dtype, heads, head_dim, page, contexts):
    import torch
    s = W.Session(W.Spec("static", dtype, *heads, head_dim, page, contexts, [1] * len(contexts), seed=76), max_ctas=64)
    s.append()
    s.attend()
    out = torch.zeros_like(s.out)
    config = pkg.GQAConfig(*heads, head_dim, s.spec.scale, s.spec.page_bytes, dtype, s.layout, s.spec.num_tokens, pkg.PLAN_BALANCED, pkg.KERNEL_AUTO, 64)
    pkg.attend_static(0, s.stream.cuda_stream, config, s.arena, s.table.page_ids_buffer(), *s.spec.batch(), s.spec.layer, s.q, out)
    s.ctx.sync()
    torch.cuda.synchronize()
    assert np.array_equal(checks.to_numpy_bits(out), checks.to_numpy_bits(s.out))
    checks.assert_attention_close(s)
    s.close()
