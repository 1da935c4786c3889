"""The froxel filter's tile edges, quotients by reciprocal and 64-bit offsets.

Without history the pass is the 3x3 mean, whose sums and quotients are IEEE-rounded in the reference's order, so it
equals the oracle bit for bit, infinities and NaN included (tolerance 0).  Volumes of 4 GB and more take the kernels
with 64-bit offsets, which compute the same as the others on the same texels (tolerance 0).
"""
import os
import sys

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import oracle  # noqa: E402
import tron_grid_gb300 as tg  # noqa: E402
from tron_grid_gb300 import fog_scene  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("whd", [(1, 1, 1), (31, 7, 7), (32, 8, 8), (33, 9, 9), (65, 17, 3)])
@pytest.mark.parametrize("f16", [True, False])
def test_mean_bit_for_bit(cuda_dev, whd, f16):
    w, h, d = whd
    rng = np.random.default_rng(w + 7 * d)
    raw = rng.exponential(1.0, (d, h, w, 4)).astype(np.float32) * 10.0 ** rng.integers(-6, 4, (d, h, w, 1))
    raw = raw.astype(np.float16 if f16 else np.float32).astype(np.float32)
    if not f16:
        raw[0, 0, 0] = [3e38, 1e-44, 0.0, 2e30]
    if w * h * d > 1:
        raw[-1, -1, -1] = [np.inf, 1.0, np.nan, 0.0]
    args = fog_scene.FogScene(fog_scene.FogSpec(width=w, height=h, depth=d)).param_args(0)
    dt = torch.float16 if f16 else torch.float32
    out = tg.fog_filter(tg.fog_params(**args), torch.from_numpy(raw).to(cuda_dev, dt),
                        torch.zeros((d, h, w, 4), dtype=dt, device=cuda_dev))
    want = oracle.fog_filter(oracle.fog_param_block(**args), raw, np.zeros_like(raw), fp16_store=f16)
    np.testing.assert_array_equal(out.float().cpu().numpy(), want)


@pytest.mark.parametrize("which", ["raw", "history"])
def test_volumes_beyond_32_bit_offsets(cuda_dev, which):
    w, h, d = 33, 9, 3
    sc = fog_scene.FogScene(fog_scene.FogSpec(width=w, height=h, depth=d), cuda_dev)
    raw, hist = sc.inject(1), sc.inject(0)
    p = tg.fog_params(**sc.param_args(1))
    want = tg.fog_filter(p, raw, hist)
    slice_elems = (1 << 31) // 2 + 64  # slices a little over 2 GB apart
    big = torch.zeros(2 * slice_elems + h * w * 4, dtype=torch.float16, device=cuda_dev)
    far = big.as_strided((d, h, w, 4), (slice_elems, w * 4, 4, 1))
    far.copy_(raw if which == "raw" else hist)
    got = tg.fog_filter(p, far if which == "raw" else raw, far if which == "history" else hist, out=torch.empty_like(raw))
    assert torch.equal(got, want)


@pytest.mark.parametrize("base", [0, (1 << 23) - 200, (1 << 24) - 200])
def test_mean_of_subnormal_sums(cuda_dev, base):
    """Boxes of six whose sums are base + 1 .. base + 408 units of 2^-149: below 2^-125 their quotients are subnormal,
    where a third of a unit and a half of one are both met.  Equals the oracle bit for bit (tolerance 0)."""
    w, h, d = 33, 9, 17
    units = np.zeros((d, h, w, 4), np.uint32)  # a float32 of these bits is that many units of 2^-149, up to 2^24
    units[:, 1::3, ::w - 1, :] = base + 1 + np.arange(d * 3 * 2 * 4, dtype=np.uint32).reshape(d, 3, 2, 4)
    raw = units.view(np.float32)
    raw[1::2] *= -1.0
    args = fog_scene.FogScene(fog_scene.FogSpec(width=w, height=h, depth=d)).param_args(0)
    out = tg.fog_filter(tg.fog_params(**args), torch.from_numpy(raw).to(cuda_dev),
                        torch.zeros((d, h, w, 4), device=cuda_dev))
    want = oracle.fog_filter(oracle.fog_param_block(**args), raw, np.zeros_like(raw), fp16_store=False)
    np.testing.assert_array_equal(out.cpu().numpy(), want)
