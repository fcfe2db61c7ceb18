"""Windows without a persistent kernel: row and column launches over chunks of
units (several angles per launch) against the per-window launches and the oracle."""
import numpy as np
import pytest

import _helpers as H
import gisspa_b200 as G
from gisspa_b200 import synth
from oracle import gisspa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from gisspa_b200 import build
    build.build_library()


# 100: many angles in one chunk; 316 = 4 79 (dense prime); 804 and 1084 with few units; 1084 with eight templates: two chunks
@pytest.mark.parametrize("l,templates", [(100, 3), (252, 4), (316, 3), (804, 5), (1084, 2), (1084, 8)])
def test_chunked_windows(l, templates):
    t = 2 * (l // 10)
    d_m = float(int(0.8 * t))
    kw = dict(apix=1.0, phi_step=90.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=d_m, thres=0.0,
              phase_flip=1, overlap=l // 4)
    ds = synth.make_dataset(40 + l, nx=int(l * 1.6), ny=int(l * 1.3) + 1, n_templates=templates, tsize=t, n_particles=2,
                            snr=0.3, n_blobs=40, ball_radius=0.3 * t, phistep=90.0, diameter=d_m, window=l,
                            overlap=l // 4, defocus=(1.0, 2.0), astig_A=300.0)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    p = O.Params(padding_size=l, **kw)
    ref = O.search(m.image, ds.templates, p, O.make_ctf(p, *ctf, l), workers=4)
    fin = np.isfinite(ref.score)
    tabs = {}
    for name in ("chunked", "timed", "graph", "per window"):
        with G.Context(0) as ctx:
            ctx.set_two_pass(name == "per window")
            ctx.set_graph(name == "graph")
            ctx.set_kernel_timing(name == "timed")
            ctx.set_templates(G.default_params(window_size=l, **kw), ds.templates, ctf)
            ctx.search(m.image, ctf)
            u = tabs[name] = ctx.units(ref.score.shape)
            if name == "timed":
                assert ctx.timings()[5] == ctx.timings()[7] >= 1 and ctx.timings()[6] > 0
        assert np.array_equal(fin, np.isfinite(u["score"])), name
        rel = np.abs(u["score"][fin] - ref.score[fin]) / np.abs(ref.score[fin])
        assert rel.max() <= H.SCORE_RTOL, (name, rel.max())
        assert np.array_equal(u["pos"][fin], ref.pos[fin]), name
    assert np.array_equal(tabs["chunked"], tabs["graph"])
