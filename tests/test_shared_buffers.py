"""Lookups whose query image shares memory with the NNF: the image is copied first, into memory the lookup
already has, so that they can be captured like any other after one lookup of the same size."""
import numpy as np
import pytest

import patchtable_b200 as ptb
from patchtable_b200 import synth
from tests.conftest import srand_all

pytestmark = pytest.mark.gpu
SIZES = [(40, 50), (33, 61)]


def _shared(n_rgb, n_ann):
    """A float64 field and an image that ends inside it, in one allocation."""
    import torch
    buf = torch.empty(n_ann * 3 + n_rgb * 3, dtype=torch.float64, device="cuda")
    ann = buf[:3 * n_ann]
    rgb = buf[3 * n_ann - 32:].view(torch.float32)[:3 * n_rgb]
    return rgb, ann


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("captured", [False, True])
def test_image_inside_the_field(gpu, libc, batched, captured):
    import torch
    pairs = [synth.pair(h, w, 30 + i) for i, (h, w) in enumerate(SIZES)]
    srand_all(libc, 1)
    t = ptb.PatchTable(ptb.PatchTableParams("-limit 0.5 -coherence_spatial 4"), pairs[0][1])
    if batched:
        qb = t.batch(SIZES)
        n_rgb, n_ann = qb.pixels, qb.patches
        img = torch.from_numpy(np.concatenate([p[0].ravel() for p in pairs])).cuda()
        call = lambda rgb, ann: qb.lookup(rgb.data_ptr(), ann.data_ptr(), torch.cuda.current_stream().cuda_stream)
    else:
        h, w = SIZES[0]
        n_rgb, n_ann = h * w, (h - 7) * (w - 7)
        img = torch.from_numpy(pairs[0][0].ravel()).cuda()
        call = lambda rgb, ann: t.lookup_device(rgb.data_ptr(), h, w, ann.data_ptr(),
                                                torch.cuda.current_stream().cuda_stream)
    want = torch.empty(3 * n_ann, dtype=torch.float64, device="cuda")
    call(img, want)                               # apart, and outside any capture
    rgb, ann = _shared(n_rgb, n_ann)
    rgb.copy_(img)
    if captured:
        held = ptb.device_bytes_in_use()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call(rgb, ann)
        assert ptb.device_bytes_in_use() == held  # nothing was allocated under capture
        rgb.copy_(img)
        g.replay()
    else:
        call(rgb, ann)
    torch.cuda.synchronize()
    assert torch.equal(ann, want)
    t.close()


def test_a_batch_holds_48_bytes_per_pixel_and_patch(gpu, libc):
    """12 bytes per pixel (the image's copy) and 36 per patch: entries, choices and states."""
    srand_all(libc, 1)
    t = ptb.PatchTable(ptb.PatchTableParams("-limit 0.5"), synth.pair(40, 50, 30)[1])
    sizes = [(400, 500), (333, 61), (8, 8)] * 3
    before = ptb.device_bytes_in_use()
    qb = t.batch(sizes)
    assert ptb.device_bytes_in_use() - before <= 12 * qb.pixels + 36 * qb.patches + 4096
    t.close()
