"""Searches where device memory holds the micrograph and its windows, but not
beside the pair spectra of many angles that the search would take ahead or that an
earlier search left."""
import numpy as np
import pytest

import gisspa_b200 as G
from gisspa_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from gisspa_b200 import build
    build.build_library()


# window 320, 12 pairs: 80 windows of a 3200 x 2560 micrograph take 65 MB and their preparation 200 MB; the pair
# spectra of the 17 angles of a launch take 167 MB, those of 72 angles 708 MB
@pytest.mark.parametrize("before,free_mb", [(False, 370), (True, 1000)])
def test_room_for_the_micrograph(before, free_mb):
    import torch
    l = 320
    kw = dict(apix=1.0, phi_step=5.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=48.0, thres=0.0,
              phase_flip=1, overlap=0)
    ds = synth.make_dataset(5, nx=400, ny=380, n_templates=24, tsize=64, n_particles=2, snr=0.3, n_blobs=40,
                            ball_radius=20.0, phistep=5.0, diameter=48.0, window=l, overlap=0, defocus=(1.0, 2.0),
                            astig_A=300.0)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    big = np.random.default_rng(2).standard_normal((2560, 3200)).astype(np.float32)
    if before:  # 262 MB for the first micrograph's successor do not fit beside 708 MB of spectra
        big = np.concatenate([big, big])  # 525 MB
    units = []
    for short in (False, True):
        held = None
        with G.Context(0) as ctx:
            ctx.set_templates(G.default_params(window_size=l, **kw), ds.templates, ctf)
            if short:
                torch.cuda.empty_cache()
                held = torch.empty(torch.cuda.mem_get_info(0)[0] - (free_mb << 20), dtype=torch.uint8, device="cuda:0")
            if before:
                ctx.search(m.image, ctf)
            ctx.search(big, ctf)
            units.append(ctx.units())
        del held
        torch.cuda.empty_cache()
    assert len(units[0]) == 72 * 24 * 80 * (2 if before else 1)
    # sums of squares are added in any order
    np.testing.assert_allclose(units[1]["score"], units[0]["score"], rtol=1e-5)


# one template and one window: a search needs some 6 and 20 MB, the default rings have 51 and 72 MB of maps
@pytest.mark.parametrize("l,free_mb", [(320, 30), (640, 50)])
def test_room_for_the_ring(l, free_mb):
    import torch
    kw = dict(apix=1.0, phi_step=30.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=20.0, thres=0.0,
              phase_flip=1, overlap=0)
    ds = synth.make_dataset(6, nx=l, ny=l, n_templates=1, tsize=24, n_particles=2, snr=0.3, n_blobs=40, ball_radius=7.0,
                            phistep=30.0, diameter=20.0, window=l, overlap=0, defocus=(1.0, 2.0), astig_A=300.0)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    units = []
    for short in (False, True):
        held = None
        with G.Context(0) as ctx:
            ctx.set_templates(G.default_params(window_size=l, **kw), ds.templates, ctf)
            if short:
                torch.cuda.empty_cache()
                held = torch.empty(torch.cuda.mem_get_info(0)[0] - (free_mb << 20), dtype=torch.uint8, device="cuda:0")
            ctx.search(m.image, ctf)
            units.append(ctx.units())
        del held
        torch.cuda.empty_cache()
    np.testing.assert_allclose(units[1]["score"], units[0]["score"], rtol=1e-5)


def test_room_for_merging():
    import torch
    n = 1000000  # 148 MB without room for pairs, 284 MB with the room that is taken first
    r = np.random.default_rng(4)
    items = np.zeros(n, G.MERGE_ITEM_DTYPE)
    items["group"] = np.arange(n) // 4
    for c in ("x", "y", "alt", "az", "phi"):
        items[c] = r.uniform(0, 20, n)
    items["score"] = r.uniform(7, 12, n)
    want = G.merge_duplicates(items, 10.0, 12.0)
    assert 0.1 * n < want.sum() < 0.95 * n
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info(0)[0] - (200 << 20), dtype=torch.uint8, device="cuda:0")
    got = G.merge_duplicates(items, 10.0, 12.0)
    del held
    torch.cuda.empty_cache()
    assert np.array_equal(got, want)
