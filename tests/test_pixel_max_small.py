"""gs_get_pixel_max of micrographs smaller than the window: the pixels on the CPU
(tests/native/test_pixmax_host.cu), the map against the oracle on a GPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import _helpers as H

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_pixels_of_the_map(tmp_path):
    exe = str(tmp_path / "test_pixmax_host")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(ROOT, "gisspa_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "test_pixmax_host.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "OK" in r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("l,nx,ny", [(160, 150, 220), (512, 400, 300), (100, 90, 99)])
def test_pixel_max_of_a_small_micrograph(l, nx, ny):
    import gisspa_b200 as G
    from gisspa_b200 import synth
    from oracle import gisspa_oracle as O
    d_m, thres = 0.2 * l, 2.5
    kw = dict(apix=1.0, phi_step=90.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=d_m, thres=thres,
              phase_flip=1, overlap=l // 4)
    ds = synth.make_dataset(7 + l, nx=3 * l, ny=3 * l, n_templates=3, tsize=l // 4, n_particles=9, snr=0.5, n_blobs=40,
                            ball_radius=l / 14, phistep=90.0, diameter=d_m, window=l, overlap=0,
                            defocus=(1.0, 2.0), astig_A=200.0)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    image = np.ascontiguousarray(m.image[l:l + ny, l:l + nx])
    with G.Context(0) as ctx:
        ctx.set_templates(G.default_params(window_size=l, **kw), ds.templates, ctf)
        ctx.search(image, ctf)
        val, tmpl, ang = ctx.pixel_max(thres, (ny, nx))
    p = O.Params(padding_size=l, **kw)
    ref = O.search(image, ds.templates, p, O.make_ctf(p, *ctf, l), workers=4, pixel_thres=thres)
    got, have = tmpl >= 0, np.isfinite(ref.pixel_value)
    assert have.sum() > 20
    tol = H.SCORE_RTOL * thres + 1e-6
    assert np.all(np.abs(val[got & ~have] - thres) <= tol)
    assert np.all(np.abs(ref.pixel_value[have & ~got] - thres) <= tol)
    both = got & have
    assert np.abs(val[both] / ref.pixel_value[both] - 1).max() <= H.SCORE_RTOL
    differ = both & ((tmpl != ref.pixel_template) | (ang != ref.pixel_angle))
    assert differ.sum() <= max(2, both.sum() // 100)
