"""The vectorised front-stage kernel at the ends of its arithmetic, against the general one on the same inputs: rows of zeros
(also with eps 0: 0 / 0), rows at the ends of their type (in f32 and bf16 with squares that overflow f32, where 1 / rms is 0, or
underflow), rows with an infinity or a NaN, and a rotation with an attention factor.  A projection that starts off a 16-byte boundary takes the general kernel."""
import numpy as np
import pytest

import checks
import gpuharness as G
import workloads as W
from oracle import psi_oracle as O

pkg = G.pkg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [pkg.F32, pkg.BF16, pkg.F16])
@pytest.mark.parametrize("eps", [0.0, 1e-6])
@pytest.mark.parametrize("yarn", [0, 1])
@pytest.mark.parametrize("runs", [[70, 60], [700, 60]])  # a step whose CTAs all fit at once, and a longer one
def test_extreme_rows_equal_the_general_kernel(dtype, eps, yarn, runs):
    import torch
    spec = W.Spec("ends", dtype, 6, 2, 128, 16, [300, 4], runs, seed=29)
    weights = [O.encode(np.linspace(0.5, 1.5, 128).astype(np.float32), O.BF16).tolist() for _ in range(2)]
    width = 2 * (6 + 2) * 128
    # (their squares lie beyond f32, or beyond it downwards; f16 ends long before: its squares are ordinary f32 values)
    big, small = (3e38, 1e-30) if dtype != pkg.F16 else (6e4, 6e-8)
    got = []
    for shift in (0, 1):
        s = W.Session(spec)
        s.gqa.set_norm_rope(pkg.NormRopeConfig(64, eps, 1e6, yarn, 4.0, 1.25, 32.0, 1.0, 8192, 1), *weights)
        torch.manual_seed(5)
        values = torch.randn((spec.num_tokens, width), device=s.device)
        values[0::8] = 0.0
        values[1::8] = big
        values[2::8] *= small
        values[3::8, ::50] = float("inf")
        values[4::8, ::70] = float("nan")
        values[5::8] = -big
        values = values.to(s.tdtype)
        held = torch.zeros(values.numel() + shift, dtype=s.tdtype, device=s.device)[shift:].view(values.shape)
        held.copy_(values)
        q, gates = torch.zeros_like(s.q), torch.zeros_like(s.q)
        s.gqa.projection_norm_rope_append(s.pages, s.table, 0, held, True, q, gates)
        s.ctx.sync()
        got.append([O.decode(checks.to_numpy_bits(x).reshape(-1), dtype).astype(np.float64) for x in (q, gates, s.arena)])
        s.close()
    # As beside the ordinary rows: the two kernels' 1 / rms differ by an ulp or two of f32 (2^-22 with the sum's order), which
    # may turn over either rounding of a normalised element to 16 bits, an ulp of it each.  A rotated output adds two of them,
    # x1 cos - x2 sin, so that two ulps of (x1, x2)'s length bound what they bring in (the rotation keeps the length, and the
    # factor is part of the outputs'), and rounds again.  Other elements have their own size for it.
    ulp = {pkg.F32: 2.0 ** -21, pkg.BF16: 2.0 ** -7, pkg.F16: 2.0 ** -10}[dtype]
    for a, b in zip(*got):
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b))
        rows = b.reshape(-1, 128)
        with np.errstate(all="ignore"):
            length = np.abs(rows)
            pair = np.tile(np.hypot(rows[:, :32], rows[:, 32:64]), 2)
        length[:, :64] = np.where(np.isfinite(pair), pair, length[:, :64])  # (a value's neighbour may be no number)
        length = length.reshape(-1)
        fine = np.isfinite(a) & np.isfinite(b)
        a, b, length = a[fine], b[fine], length[fine]
        near = np.abs(b) < 1e4  # (gates and values pass through with the inputs' size: those are equal)
        assert np.array_equal(a[~near], b[~near])
        a, b, length = a[near], b[near], length[near]
        assert np.all(np.abs(a - b) <= 2 * ulp * length + ulp * np.abs(b))
