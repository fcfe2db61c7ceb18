"""norm_type 1 on the persistent kernel against the per-window passes and the
oracle: blocks of several rows, of parts of rows and straddling rows, odd
template counts, several angle groups."""
import numpy as np
import pytest

import gisspa_b200 as G
from gisspa_b200 import synth
from oracle import gisspa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from gisspa_b200 import build
    build.build_library()


def _key(p):
    """A pick's unit and 1024-element block cannot be told apart from its position alone: unit and centre."""
    return (int(p["angle_index"]), int(p["window_x"]), int(p["window_y"]), int(p["template_index"]),
            float(p["center_x"]), float(p["center_y"]))


@pytest.mark.parametrize("l,templates", [(96, 3), (128, 4), (224, 3), (320, 5), (352, 2), (512, 3), (640, 3)])
def test_norm1_windows(l, templates):
    t = 2 * (l // 8)
    kw = dict(apix=1.0, phi_step=45.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=float(int(0.8 * t)),
              thres=3.0, phase_flip=1, overlap=l // 4, norm_type=1)
    ds = synth.make_dataset(70 + l, nx=int(l * 1.5), ny=int(l * 1.2) + 1, n_templates=templates, tsize=t, n_particles=2,
                            snr=0.3, n_blobs=40, ball_radius=0.3 * t, phistep=45.0, diameter=kw["d_m"], window=l,
                            overlap=l // 4, defocus=(1.0, 2.0), astig_A=300.0)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    got = {}
    for name in ("persistent", "passes", "one angle per launch"):
        with G.Context(0) as ctx:
            ctx.set_two_pass(name == "passes")
            ctx.set_angles_per_launch(1 if name == "one angle per launch" else 0)
            ctx.set_templates(G.default_params(window_size=l, **kw), ds.templates, ctf)
            got[name] = ctx.search(m.image, ctf)
    p = O.Params(padding_size=l, **kw)
    ref, _, _ = O.search_norm1(m.image, ds.templates, p, O.make_ctf(p, *ctf, l))
    want = {(q.angle_index, q.window_i, q.window_j, q.template, q.cx, q.cy): q.score for q in ref}
    assert len(want) > 20
    for name, picks in got.items():
        have = {_key(q): float(q["score"]) for q in picks}
        assert len(have) == len(picks)
        # z rounds at 2e-5: picks may differ only that close to the threshold, or where two values of a block tie
        close = [k for k in set(want) ^ set(have) if abs(want.get(k, have.get(k)) - 3.0) > 2e-4]
        assert len(close) <= len(want) // 500, (name, close[:4])
        both = [(want[k], have[k]) for k in set(want) & set(have)]
        assert max(abs(a - b) / abs(a) for a, b in both) < 1e-4, name
        order = [tuple(int(q[c]) for c in ("angle_index", "window_y", "window_x", "template_index")) for q in picks]
        assert order == sorted(order), name
