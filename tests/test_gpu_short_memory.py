"""Searches on a device with little free memory: launches of fewer angles, the same results."""
import numpy as np
import pytest

import gisspa_b200 as G
from gisspa_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from gisspa_b200 import build
    build.build_library()


# chunked launches, the persistent kernel (with and without a graph), norm_type 1: 72 angles of 12 pair spectra are
# 0.6 to 0.7 GB, 0.5 GB are free
@pytest.mark.parametrize("l,norm_type,graph", [(300, 0, False), (320, 0, False), (320, 0, True), (320, 1, False)])
def test_short_memory(l, norm_type, graph):
    import torch
    kw = dict(apix=1.0, phi_step=5.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=48.0,
              thres=4.5 if norm_type else 0.0, phase_flip=1, overlap=l // 4, norm_type=norm_type)
    ds = synth.make_dataset(90 + l, nx=int(l * 1.5), ny=int(l * 1.2) + 1, n_templates=24, tsize=64, n_particles=2,
                            snr=0.3, n_blobs=40, ball_radius=20.0, phistep=5.0, diameter=48.0, window=l,
                            overlap=l // 4, defocus=(1.0, 2.0), astig_A=300.0)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    got = []
    for short in (False, True):
        held = None
        with G.Context(0) as ctx:
            ctx.set_angles_per_launch(72)
            ctx.set_graph(graph)
            ctx.set_templates(G.default_params(window_size=l, **kw), ds.templates, ctf)
            if short:
                torch.cuda.empty_cache()
                held = torch.empty(torch.cuda.mem_get_info(0)[0] - (1 << 29), dtype=torch.uint8, device="cuda:0")
            for _ in range(2):  # the second on the buffers of the first
                got.append(ctx.search(m.image, ctf))
        del held
        torch.cuda.empty_cache()
    want = {tuple(int(p[c]) for c in ("angle_index", "window_y", "window_x", "template_index", "center_x", "center_y")):
            float(p["score"]) for p in got[0]}
    assert len(want) > 20
    for picks in got[1:]:
        have = {tuple(int(p[c]) for c in ("angle_index", "window_y", "window_x", "template_index", "center_x",
                                          "center_y")): float(p["score"]) for p in picks}
        # sums in another order: scores within a few float roundings, z-scores (float sums over 1728 maps) within 2e-5
        # of the threshold's side
        both = want.keys() & have.keys()
        assert all(abs(want[k] - have[k]) <= 1e-4 * abs(want[k]) for k in both)
        assert all(abs(d.get(k, 4.5) - 4.5) <= 1e-3 for d in (want, have) for k in d.keys() - both)
