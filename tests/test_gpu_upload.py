"""Micrograph uploads: pageable memory above and below the size that is staged
by threads, pinned memory, device memory, and batches that reuse both input
buffers with sizes that change, all give the same picks."""
import numpy as np
import pytest

import gisspa_b200 as G
from gisspa_b200 import synth

pytestmark = pytest.mark.gpu


def test_uploads_give_the_same_picks():
    torch = pytest.importorskip("torch")
    from gisspa_b200 import build
    build.build_library()
    sizes = [(2048, 1530), (500, 400), (1600, 1311), (1024, 1023), (1024, 1024), (2048, 1536)]
    ds = synth.make_dataset(5, nx=512, ny=512, sizes=sizes, n_micrographs=len(sizes), n_templates=3, tsize=64, n_particles=4,
                            snr=0.5, n_blobs=40, ball_radius=20.0, phistep=90.0, diameter=48.0, window=128, overlap=32)
    gp = G.default_params(apix=1.0, phi_step=90.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=48.0,
                          thres=6.0, window_size=128, overlap=32, phase_flip=1)
    ctfs = [(m.defocus, m.dfdiff, m.dfang) for m in ds.micrographs]
    with G.Context(0) as ctx:
        ctx.set_templates(gp, ds.templates, ctfs[0])
        want = []
        for m, c in zip(ds.micrographs, ctfs):
            d = torch.from_numpy(m.image).cuda()
            want.append(ctx.search_device(d.data_ptr(), m.image.shape[1], m.image.shape[0], c))
            pinned = torch.from_numpy(m.image).pin_memory().numpy()
            assert np.array_equal(ctx.search(m.image.copy(), c), want[-1])
            assert np.array_equal(ctx.search(pinned, c), want[-1])
        assert sum(len(w) for w in want) > 5
        # (the first 64 MiB are not staged)
        for order in (range(len(sizes)), range(len(sizes)), reversed(range(len(sizes)))):
            order = list(order)
            got = ctx.search_batch([ds.micrographs[k].image for k in order], [ctfs[k] for k in order])
            for g, k in zip(got, order):
                assert np.array_equal(g, want[k])
