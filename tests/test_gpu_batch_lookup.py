"""The stage kernels' stream lookup: one-pixel streams (a tile each), more than 32 and more than 256 of them, and the
last tiles of wide strides, against single handles.  The kernels are the same, so the bits are (tolerance 0).
"""
import os
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import tron_grid_gb300 as tg  # noqa: E402
from tron_grid_gb300 import scene  # noqa: E402
from tron_grid_gb300.batch import Batch  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,pick", [([(1, 1)] * 33 + [(70, 41)], None),
                                        ([(33 + k % 3, 9) for k in range(64)] + [(301, 97)], range(0, 65, 2)),
                                        ([(17, 5 + k % 4) for k in range(257)], range(250, 257))])
def test_streams_match_handles(cuda_dev, sizes, pick):
    ids = list(range(len(sizes))) if pick is None else list(pick)
    b = Batch(sizes, storage=tg.STORAGE_FP32)
    dens = {k: tg.Denoiser(*sizes[k]) for k in ids}
    scenes = {k: scene.PlaneScene(scene.pan_with_disocclusion(*sizes[k], seed=k), cuda_dev) for k in ids}
    for t in (29, 30):
        fr = [{q: v for q, v in scenes[k].frame(t).items() if q in ("radiance", "depth", "normal", "motion")} for k in ids]
        outs = [torch.empty((sizes[k][1], sizes[k][0], 4), device=cuda_dev) for k in ids]
        b.denoise(ids, fr, outs)
        b.synchronize()
        for k, f, o in zip(ids, fr, outs):
            assert torch.equal(dens[k].denoise(**f), o)
    b.close()
    for d in dens.values():
        d.close()


@pytest.mark.parametrize("n", [256, 257])
def test_lookup_over_many_streams(cuda_dev, n):
    """A step of 256 streams is the last that looks a tile's stream up by ballots; one of 257 searches by halves."""
    sizes = [(17 + k % 40, 5 + k % 4) for k in range(n)]
    b = Batch(sizes, storage=tg.STORAGE_FP32)
    picks = [0, 31, 32, 33, 128, 254, n - 1]
    dens = {k: tg.Denoiser(*sizes[k]) for k in picks}
    scenes = [scene.PlaneScene(scene.pan_with_disocclusion(*s, seed=k), cuda_dev) for k, s in enumerate(sizes)]
    for t in (29, 30):
        fr = [{q: v for q, v in sc.frame(t).items() if q in ("radiance", "depth", "normal", "motion")} for sc in scenes]
        outs = [torch.empty((h, w, 4), device=cuda_dev) for w, h in sizes]
        b.denoise(list(range(n)), fr, outs)
        b.synchronize()
        for k in picks:
            assert torch.equal(dens[k].denoise(**fr[k]), outs[k])
    b.close()
    for d in dens.values():
        d.close()
