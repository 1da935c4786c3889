"""The spatial variance estimate of single streams (small frames: a CTA per flagged block; others, here 1282x730: two
pixels per thread over listed blocks) against the persistent batch kernel (one pixel per thread over flagged blocks):
equal bits (tolerance 0).

The first frames after a cut take the estimate everywhere; sizes leave remainders of the 32 x 4 blocks.
"""
import os
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import tron_grid_gb300 as tg  # noqa: E402
from tron_grid_gb300 import _lib as L  # noqa: E402
from tron_grid_gb300 import scene  # noqa: E402
from tron_grid_gb300.batch import Batch  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [False, True])
def test_list_equals_flags(cuda_dev, half):
    sizes = [(1, 1), (31, 3), (33, 5), (70, 7), (64, 130), (577, 290), (1282, 730)]
    st = tg.STORAGE_FP16 if half else tg.STORAGE_FP32
    b = Batch(sizes, storage=st, strategy=L.BATCH_PERSISTENT)
    dens = [tg.Denoiser(w, h, storage=st) for w, h in sizes]
    scenes = [scene.PlaneScene(scene.pan_with_disocclusion(w, h, seed=k), cuda_dev) for k, (w, h) in enumerate(sizes)]
    for t in (28, 29, 30, 31, 29):
        fr = []
        for sc in scenes:
            f = sc.frame(t)
            d = {k: f[k] for k in ("radiance", "depth", "normal", "motion")}
            if half:
                d["radiance"] = d["radiance"].half()
                d["normal"] = scene.oct16_encode(d["normal"]).contiguous()
            fr.append(d)
        outs = [torch.empty((h, w, 4), device=cuda_dev) for w, h in sizes]
        b.denoise(list(range(len(sizes))), fr, outs)
        b.synchronize()
        for d, f, o in zip(dens, fr, outs):
            assert torch.equal(d.denoise(**f), o)
    b.close()
    for d in dens:
        d.close()
