"""Persistent correlation at windows l = 16 N2 beyond 512, 720 and 768: the
smallest, odd N2 (prime-factor transforms), prime factors 7 to 23, register
limits, both tile widths, against the oracle per unit."""
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


@pytest.mark.parametrize("l", [96, 112, 160, 176, 256, 272, 304, 320, 336, 368, 400, 432, 560, 576, 592, 624, 640, 736])
def test_window_matches_oracle(l):
    t = 2 * (l // 8)
    d_m = float(int(0.8 * t))
    kw = dict(apix=1.0, phi_step=120.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=d_m, thres=0.0,
              phase_flip=1, overlap=l // 4)
    ds = synth.make_dataset(40 + l, nx=int(l * 1.6), ny=int(l * 1.3) + 1, n_templates=3, tsize=t, n_particles=2, snr=0.3,
                            n_blobs=40, ball_radius=0.3 * t, phistep=120.0, diameter=d_m, window=l, overlap=l // 4,
                            defocus=(1.0, 2.0), astig_A=300.0)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    p = O.Params(padding_size=l, **kw)
    ref = O.search(m.image, ds.templates, p, O.make_ctf(p, *ctf, l), workers=4)
    fin = np.isfinite(ref.score)
    for tile in (16, 8):
        with G.Context(0) as ctx:
            ctx.set_corr_tile(tile)
            ctx.set_templates(G.default_params(window_size=l, **kw), ds.templates, ctf)
            ctx.search(m.image, ctf)
            u = ctx.units(ref.score.shape)
            assert ctx.tuning()[4] == tile
        assert np.array_equal(fin, np.isfinite(u["score"]))
        rel = np.abs(u["score"][fin] - ref.score[fin]) / np.abs(ref.score[fin])
        assert rel.max() <= H.SCORE_RTOL, rel.max()
        assert np.array_equal(u["pos"][fin], ref.pos[fin])


def test_tensor_core_modes_stay_with_their_windows():
    """The tensor-core modes are refused at windows that only the FP32 kernel covers."""
    rng = np.random.default_rng(0)
    for precision in (G.GS_PREC_TC_BF16, G.GS_PREC_TC_FP16, G.GS_PREC_TC_FULL):
        with G.Context(0) as ctx:
            p = G.default_params(apix=1.0, phi_step=180.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0,
                                 d_m=60.0, window_size=320, overlap=64, phase_flip=1, precision=precision)
            ctx.set_templates(p, rng.standard_normal((2, 64, 64)).astype(np.float32), (1.5, 0.0, 0.0))
            with pytest.raises(G.GisspaError) as e:
                ctx.search(rng.standard_normal((400, 400)).astype(np.float32), (1.5, 0.0, 0.0))
            assert e.value.status == G.GS_ERR_UNSUPPORTED


def test_autotuner_at_a_small_window():
    """The ring that the window's own rule takes is larger than the tuner's candidates."""
    ds = synth.make_dataset(3, nx=500, ny=400, n_templates=5, tsize=48, n_particles=2, snr=0.3, n_blobs=40,
                            ball_radius=15.0, phistep=60.0, diameter=36.0, window=128, overlap=32)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    tabs = []
    for tune in (False, True):
        with G.Context(0) as ctx:
            ctx.set_autotune(tune)
            ctx.set_templates(G.default_params(apix=1.0, phi_step=60.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0,
                                               lowres=100.0, d_m=36.0, window_size=128, overlap=32, phase_flip=1),
                              ds.templates, ctf)
            ctx.search(m.image, ctf)
            tabs.append(ctx.units())
    assert np.array_equal(tabs[0]["pos"], tabs[1]["pos"])
    assert np.allclose(tabs[0]["score"], tabs[1]["score"], rtol=1e-6, equal_nan=True)
