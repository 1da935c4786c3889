"""The bloom / post chain's shared work: pixel pairs, 2x2 upsample blocks, unaligned images, the corners' samples.

Bloom mips equal the oracle's bit for bit; display bytes are within one unit of it and at least 99.9% identical (the
sRGB power is CUDA's).  An image at an odd offset or pitch takes the scalar loads and stores, which give the same
bytes as the wide ones (tolerance 0).
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

pytestmark = pytest.mark.gpu


def hdr(w, h):
    rng = np.random.default_rng(w * 3 + h)
    a = rng.exponential(1.0, (h, w, 4)).astype(np.float32) * rng.choice([0.3, 8.0], (h, w, 1))
    return a.astype(np.float16).astype(np.float32)


# 3000 wide: the outer corners sample a pixel away from their own; odd sizes: clamped blocks at every mip
@pytest.mark.parametrize("wh", [(1, 2), (2, 1), (3, 3), (65, 33), (127, 130), (3000, 40)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_chain_against_oracle(cuda_dev, wh, dtype):
    w, h = wh
    img = hdr(w, h)
    if w > 64:
        img[5, 7, 0] = np.inf
    if dtype == torch.float32 and w > 64:
        img[20, 40, :3] = [3e38, 1.0, 2.0]
    pp = tg.PostProcessor(w, h)
    got = pp.process(torch.from_numpy(img).to(cuda_dev, dtype), order="rgba").cpu().numpy().astype(np.int32)
    want, mips = oracle.post_frame(img)
    for k, m in enumerate(pp.bloom_mips()):
        np.testing.assert_array_equal(m[..., :3], np.asarray(mips[k], np.float32)[..., :3], err_msg=f"mip {k}")
    d = np.abs(got - np.rint(np.nan_to_num(want) * 255).astype(np.int32))
    assert d.max() <= 1 and (d == 0).mean() >= 0.999
    pp.close()


@pytest.mark.parametrize("order", ["bgra", "rgba"])
def test_unaligned_images_give_the_same_bytes(cuda_dev, order):
    w, h = 70, 33
    img = torch.from_numpy(hdr(w, h)).to(cuda_dev, torch.float16)
    pp = tg.PostProcessor(w, h)
    want = pp.process(img, order=order).clone()
    src = torch.zeros(h * (w + 1) * 4 + 4, dtype=torch.float16, device=cuda_dev)[4:].as_strided((h, w, 4), ((w + 1) * 4, 4, 1))
    src.copy_(img)
    dst = torch.zeros(h * (w + 1) * 4 + 4, dtype=torch.uint8, device=cuda_dev)[4:].as_strided((h, w, 4), ((w + 1) * 4, 4, 1))
    pp.process(src, dst, order=order)
    assert torch.equal(dst, want)
    pp.close()
