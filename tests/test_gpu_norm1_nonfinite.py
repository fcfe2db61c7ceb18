"""norm_type 1 on maps that are not finite, zero or overflow their squares:
the persistent kernel's block maxima and picks are those of the per-window
passes (z = 0 where the deviation is not positive)."""
import os
import subprocess

import numpy as np
import pytest

import gisspa_b200 as G
from gisspa_b200 import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from gisspa_b200 import build
    build.build_library()


@pytest.mark.parametrize("l", [96, 352])
@pytest.mark.parametrize("what", ["nan pixel", "infinite pixel", "nan template", "zero", "overflow"])
def test_norm1_not_finite(l, what):
    kw = dict(apix=1.0, phi_step=90.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=20.0,
              thres=-1.0, phase_flip=0, overlap=l // 4, norm_type=1)
    ds = synth.make_dataset(30 + l, nx=int(l * 1.5), ny=int(l * 1.2), n_templates=3, tsize=24, n_particles=2,
                            snr=0.3, n_blobs=40, ball_radius=7.0, phistep=90.0, diameter=20.0, window=l,
                            overlap=l // 4, defocus=(1.0, 2.0), astig_A=300.0)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    img, tmpl = m.image.copy(), ds.templates.copy()
    if what == "nan pixel":
        img[10, 20] = np.nan
    elif what == "infinite pixel":
        img[10, 20] = np.inf
    elif what == "nan template":
        tmpl[1, 3, 4] = np.nan
    elif what == "zero":
        img[:] = 0.0
    else:
        # maps / l^2 around 1e20: their squares overflow, and the squares of their means at some of the pixels.
        # (the offset keeps the hot-pixel clamp off)
        img += np.float32(10.0)
        with G.Context(0) as ctx:
            ctx.set_templates(G.default_params(window_size=l, **dict(kw, norm_type=0)), tmpl, ctf)
            ctx.search(img, ctf)
            img *= np.float32(1e20 * l * l / np.median(ctx.units()["sigma"]))
    got = []
    for passes in (True, False):
        with G.Context(0) as ctx:
            ctx.set_two_pass(passes)
            ctx.set_templates(G.default_params(window_size=l, **kw), tmpl, ctf)
            got.append(ctx.search(img, ctf))
    want, have = got
    assert len(want) > 100
    for c in ("angle_index", "window_x", "window_y", "template_index", "center_x", "center_y", "score"):
        assert np.array_equal(want[c], have[c]), c


def test_reciprocal_deviation(tmp_path):
    """tests/native/test_norm1_moments.cu"""
    exe = str(tmp_path / "test_norm1_moments")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(ROOT, "gisspa_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "test_norm1_moments.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "OK" in r.stdout
