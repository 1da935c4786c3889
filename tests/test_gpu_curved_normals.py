"""FP16 storage where every pixel's octahedral code differs from its neighbours' (no flat surfaces).

The temporal pass decodes normals only where a tap's code differs from the pixel's; here all do.  Tolerance as for the
FP16 form elsewhere: within 2^-8 per pixel and 1e-4 on average of the float32 oracle that rounds the same stores.
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
from tron_grid_gb300 import scene  # noqa: E402
from tests.helpers import rel_err  # noqa: E402

pytestmark = pytest.mark.gpu


def test_curved_normals_fp16(cuda_dev):
    w, h = 131, 67
    sc = scene.PlaneScene(scene.pan_with_disocclusion(w, h, seed=9))
    den = tg.Denoiser(w, h, storage=tg.STORAGE_FP16)
    st = oracle.FullState(h, w, np.float32)
    params = oracle.full_params()
    yy, xx = np.mgrid[0:h, 0:w].astype(np.float32)
    for t in range(5):
        f = sc.frame(28 + t)
        # a bumpy surface that moves by about a pixel a frame: some taps pass the normal test, some fail it
        n = np.stack([np.sin(0.11 * (xx + t)), np.cos(0.17 * yy), 1.1 + np.sin(0.05 * (xx - yy))], -1)
        n /= np.linalg.norm(n, axis=-1, keepdims=True)
        enc = scene.oct16_encode(torch.from_numpy(n.astype(np.float32))).contiguous()
        rad = f["radiance"].half()
        out = torch.empty((h, w, 4), dtype=torch.float16, device=cuda_dev)
        den.denoise(rad.to(cuda_dev), f["depth"].to(cuda_dev), enc.to(cuda_dev), f["motion"].to(cuda_dev), out=out)
        want, _ = oracle.full_frame(params, st, rad.float().numpy(), f["depth"].numpy(), oracle.oct16_decode(enc.numpy()),
                                    f["motion"].numpy(), fp16_store=oracle.fp16_storage_mask(True))
        e = rel_err(out.float().cpu().numpy(), want)
        assert e.max() <= 2.0 ** -8 and e.mean() <= 1e-4, f"frame {t}: max {e.max():.2e}, mean {e.mean():.2e}"
    den.close()
