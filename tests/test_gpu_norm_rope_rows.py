"""The vectorised front-stage kernel against the general one on the same inputs: a projection that starts off a 16-byte
boundary takes the general kernel, an aligned copy of it the vectorised one."""
import numpy as np
import pytest

import checks
import gpuharness as G
import workloads as W
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [pkg.F32, pkg.BF16, pkg.F16])
@pytest.mark.parametrize("heads,head_dim,rope_dim", [((5, 1), 64, 16), ((24, 4), 256, 64), ((40, 8), 128, 128), ((16, 2), 256, 96),
                                                     ((3, 3), 128, 48)])
@pytest.mark.parametrize("runs", [[1], [3, 1, 20, 2], [900, 1, 700]])
def test_vectorised_rows_equal_the_general_kernel(dtype, heads, head_dim, rope_dim, runs):
    import torch
    rng = np.random.default_rng(head_dim + rope_dim)
    spec = W.Spec("rows", dtype, *heads, head_dim, 16, [300, 41, 0, 1000][:len(runs)], runs, seed=23)
    weights = [O.encode(1.0 + 0.1 * rng.standard_normal(head_dim).astype(np.float32), O.BF16).tolist() for _ in range(2)]
    width = 2 * (heads[0] + heads[1]) * head_dim
    got = []
    for shift in (0, 1):
        s = W.Session(spec)
        s.gqa.set_norm_rope(pkg.NormRopeConfig(rope_dim, 1e-6, 1e6, 0, 1, 1, 1, 1, 1, 0), *weights)
        if shift == 0:
            torch.manual_seed(head_dim + rope_dim)
            values = torch.randn((spec.num_tokens, width), device=s.device).to(s.tdtype)
        held = torch.zeros(values.numel() + shift, dtype=s.tdtype, device=s.device)[shift:].view(values.shape)
        held.copy_(values)
        q, gates = torch.zeros_like(s.q), torch.zeros_like(s.q)
        s.gqa.projection_norm_rope_append(s.pages, s.table, 0, held, True, q, gates)
        s.ctx.sync()
        got.append([checks.to_numpy_bits(x) for x in (q, gates, s.arena)])
        s.close()
    (q0, g0, a0), (q1, g1, a1) = got
    assert np.array_equal(g0, g1)
    # The two kernels sum a row's squares in another order, which moves 1 / rms by an ulp of f32.  In 16 bits that may turn
    # over either of the two roundings of a normalised element, one ulp of it each; a rotated output adds two such elements
    # (|c| + |s| <= sqrt(2)), each at most `top` in magnitude, and rounds once more.
    ulp = {pkg.F32: 2.0 ** -22, pkg.BF16: 2.0 ** -7, pkg.F16: 2.0 ** -10}[dtype]
    for a, b in ((q0, q1), (a0, a1)):
        a, b = (O.decode(x.reshape(-1), dtype).astype(np.float64) for x in (a, b))
        top = np.abs(b).max() * 2 ** 0.5
        assert np.all(np.abs(a - b) <= 2 * ulp * 2 ** 0.5 * top + ulp * np.abs(b))
        if dtype != pkg.F32:
            assert np.mean(a == b) > 0.98
