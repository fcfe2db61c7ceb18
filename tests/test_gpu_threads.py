"""Host threads with a context each on one GPU: searches whose transforms take
different amounts of shared memory do not disturb one another."""
import threading

import numpy as np
import pytest

import gisspa_b200 as G
from gisspa_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from gisspa_b200 import build
    build.build_library()


@pytest.mark.parametrize("generic", [False, True])
def test_contexts_in_two_threads(generic):
    l = 96
    kw = dict(apix=1.0, phi_step=180.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=100.0, d_m=20.0, thres=4.0,
              phase_flip=1, overlap=0)
    ds = synth.make_dataset(17, nx=200, ny=180, n_templates=2, tsize=24, n_particles=2, snr=0.3, n_blobs=40,
                            ball_radius=7.0, phistep=180.0, diameter=20.0, window=l, overlap=0, defocus=(1.0, 2.0),
                            astig_A=300.0)
    m = ds.micrographs[0]
    ctf = (m.defocus, m.dfdiff, m.dfang)
    # rows of 100 and of 5760 pixels: more and less shared memory per CTA than the default limit
    images = [m.image[:100, :100].copy(), np.random.default_rng(1).standard_normal((96, 5760)).astype(np.float32)]
    errors, results = [], [[] for _ in range(16)]

    def work(k):
        try:
            with G.Context(0) as ctx:
                ctx.set_generic_fft(generic)
                ctx.set_templates(G.default_params(window_size=l, **kw), ds.templates, ctf)
                for _ in range(500):
                    ctx.search(images[k % 2], ctf)
                results[k] = ctx.units()["score"].copy()
        except Exception as e:  # noqa: BLE001
            errors.append((k, str(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(16)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(2, 16):
        # sums of squares are added in any order
        np.testing.assert_allclose(results[k], results[k % 2], rtol=1e-5)
