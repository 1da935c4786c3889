"""The a-trous kernels of one, two and three output rows per thread compute the same: equal bits (tolerance 0).

FULL: the TMA kernels (one row for small frames, two at 385x211, three at the last level of others and at every level
of a large frame) against the plain-load kernels (two rows).  REF_EXACT: the handle's chain (three rows from about
0.6 Mpx) against the chain of the entry point without allocation (two rows).  Sizes leave remainders of the 12- and
8-row tiles and of the residue planes.
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
from tron_grid_gb300 import _lib as L  # noqa: E402
from tron_grid_gb300 import scene  # noqa: E402
from tron_grid_gb300.svgf import image  # noqa: E402
from tests.helpers import REL_TOL, rel_err  # noqa: E402

pytestmark = pytest.mark.gpu


def frames(w, h, half, n, dev):
    sc = scene.PlaneScene(scene.pan_with_disocclusion(w, h, seed=w), dev)
    for t in range(n):
        f = sc.frame(29 + t)
        d = {k: f[k] for k in ("radiance", "depth", "normal", "motion")}
        if half:
            d["radiance"] = d["radiance"].half()
            d["normal"] = scene.oct16_encode(d["normal"]).contiguous()
        yield d


@pytest.mark.parametrize("wh", [(1, 1), (33, 13), (70, 25), (96, 61), (385, 211), (640, 361), (3842, 1213)])
@pytest.mark.parametrize("half", [False, True])
def test_full_rows(cuda_dev, wh, half):
    w, h = wh
    st = tg.STORAGE_FP16 if half else tg.STORAGE_FP32
    a = tg.Denoiser(w, h, storage=st)
    b = tg.Denoiser(w, h, storage=st, flags=L.FLAG_NO_TMA)
    for f in frames(w, h, half, 3, cuda_dev):
        x, y = a.denoise(**f), b.denoise(**f)
        assert torch.equal(x, y)
    a.close()
    b.close()


@pytest.mark.parametrize("levels", [1, 2, 6])
def test_full_rows_other_level_counts(cuda_dev, levels):
    a = tg.Denoiser(200, 77, levels=levels)
    b = tg.Denoiser(200, 77, levels=levels, flags=L.FLAG_NO_TMA)
    for f in frames(200, 77, False, 2, cuda_dev):
        assert torch.equal(a.denoise(**f), b.denoise(**f))
    a.close()
    b.close()


@pytest.mark.parametrize("wh,half", [((1023, 601), True), ((1280, 720), True), ((961, 539), False)])
def test_ref_rows(cuda_dev, wh, half):
    w, h = wh
    dt = torch.float16 if half else torch.float32
    den = tg.Denoiser(w, h, mode=tg.MODE_REF_EXACT, storage=tg.STORAGE_FP16 if half else tg.STORAGE_FP32)
    p = L.default_params(tg.MODE_REF_EXACT, tg.STORAGE_FP16 if half else tg.STORAGE_FP32)
    mom = [torch.zeros((h, w, 2), dtype=dt, device=cuda_dev) for _ in range(2)]
    mimg = [L.Image(m.data_ptr(), 0, L.FMT_RG16F if half else L.FMT_RG32F, 0) for m in mom]
    for t, f in enumerate(frames(w, h, half, 2, cuda_dev)):
        want = torch.empty((h, w, 4), dtype=dt, device=cuda_dev)
        raw, out = image("radiance", f["radiance"]), image("denoised", want)
        L.check(L.load().tg_svgf_denoise_ref_noalloc(p, w, h, raw, mimg[t & 1], mimg[(t & 1) ^ 1], out,
                                                     torch.cuda.current_stream().cuda_stream))
        got = den.denoise(f["radiance"], out=torch.empty_like(want))
        assert torch.equal(got, want)
    den.close()


@pytest.mark.parametrize("wh", [(1281, 721), (1284, 723)])
@pytest.mark.parametrize("half", [False, True])
def test_ref_three_rows(cuda_dev, wh, half):
    """Chains of three rows (10 * 152 tiles of 32 x 12 and more) in both storage forms: staged by TMA and by plain loads
    the bits are equal, and equal to the oracle's within the parity tests' tolerance (binary16 images: one step of the
    store in each of the three passes, 2^-10 relative each)."""
    w, h = wh
    assert ((w + 31) // 32) * ((h + 11) // 12) >= 10 * 152
    st, dt = (tg.STORAGE_FP16, torch.float16) if half else (tg.STORAGE_FP32, torch.float32)
    a = tg.Denoiser(w, h, mode=tg.MODE_REF_EXACT, storage=st)
    b = tg.Denoiser(w, h, mode=tg.MODE_REF_EXACT, storage=st, flags=L.FLAG_NO_TMA)
    mom = np.zeros((h, w, 2), np.float32)
    for f in frames(w, h, half, 2, cuda_dev):
        x, y = (d.denoise(f["radiance"], out=torch.empty((h, w, 4), dtype=dt, device=cuda_dev)) for d in (a, b))
        assert torch.equal(x, y)
        want, mom = oracle.ref_frame(f["radiance"].float().cpu().numpy(), mom, fp16_store=half)
        assert rel_err(x.float().cpu().numpy(), want).max() <= (3 * 2.0 ** -10 if half else REL_TOL)
    a.close()
    b.close()
