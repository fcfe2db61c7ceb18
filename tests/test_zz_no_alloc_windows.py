"""gs_correlate_window_noalloc on its three routes (persistent kernel with and
without reuse of the ring, planned transforms, the two-pass kernels of window
720) against float64 maps, also under stream capture."""
import numpy as np
import pytest

import _helpers as H
import gisspa_b200 as G

pytestmark = pytest.mark.gpu


def _reference(W, P, n, d_m):
    import torch
    l = W.shape[-1]
    q = float(np.float32(d_m) / np.float32(4))
    k = torch.arange(l, device=W.device).double()
    keep = (k >= q) & (k <= l - q)
    out = []
    for p in P:
        s = torch.fft.ifft2(W.to(torch.complex128) * p.to(torch.complex128).conj(), norm="forward")
        s = s.roll((l // 2, l // 2), (0, 1)) * (1.0 if (l // 2) % 2 == 0 else -1.0)
        for m in (s.real, s.imag):
            flat = m.reshape(-1)
            peak, pos = torch.where(keep[:, None] & keep[None, :], m, torch.zeros_like(m)).reshape(-1).max(0)
            rc = float(l * l - 1)
            sd = torch.sqrt((flat.square().sum() - peak * peak) / rc - ((flat.sum() - peak) / rc) ** 2)
            out.append((float(peak / sd), int(pos)))
    return out[:n]


@pytest.mark.parametrize("l,n", [(96, 1), (160, 700), (320, 9), (512, 41), (576, 30), (768, 26), (720, 5), (300, 7), (202, 3), (1000, 12), (400, 4)])
def test_noalloc_routes(l, n):
    torch = pytest.importorskip("torch")
    from gisspa_b200 import build
    build.build_library()
    g = torch.Generator(device="cuda").manual_seed(l)
    d_m = l * 0.2
    # white windows and smooth templates with a mean, so that the maps' sums matter too
    win = torch.randn(l, l, generator=g, device="cuda", dtype=torch.float64) + 0.1
    t = torch.randn(2 * ((n + 1) // 2), l, l, generator=g, device="cuda", dtype=torch.float64)
    W = (torch.fft.fft2(win) / (l * l)).to(torch.complex64)
    T = torch.fft.fft2(t) / (l * l)
    if n % 2:
        T[-1] = 0
    P = (T[0::2] - 1j * T[1::2]).to(torch.complex64).contiguous()
    want = _reference(W, P, n, d_m)
    units = torch.full((n + 1, 4), float("nan"), device="cuda")

    def call():
        G.correlate_window_noalloc(W.data_ptr(), P.data_ptr(), n, l, d_m, units.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)

    def check():
        got = units.cpu().numpy()
        assert np.isnan(got[n]).all()  # nothing behind the last template
        pos = got[:, 1].copy().view(np.int32)
        for j, (score, at) in enumerate(want):
            assert abs(got[j, 0] - score) <= H.SCORE_RTOL * abs(score), (j, got[j], score)
            assert pos[j] == at, (j, pos[j], at)

    for _ in range(2):
        units.fill_(float("nan"))
        call()
        check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    units.fill_(float("nan"))
    graph.replay()
    check()
