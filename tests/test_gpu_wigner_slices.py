"""SO(3) transforms on both sides of the choice where a slice's low orders run (following in the
slice's stream, or beside it), against one spin transform per slice, and replayed from a graph."""

import numpy as np
import pytest

import oracle
from tests.conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def s2b():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import s2fft_b200

    return s2fft_b200


@pytest.mark.parametrize("L,N,reality", [(127, 2, False), (128, 2, False), (159, 3, False),
                                         (160, 3, False), (160, 4, False), (160, 5, False),
                                         (160, 6, False), (256, 6, False), (160, 5, True),
                                         (160, 6, True)])
@pytest.mark.parametrize("sampling", ["mw", "gl"])
def test_slices_against_spin_transforms(s2b, rng, sampling, L, N, reality):
    import torch

    flmn = torch.tensor(oracle.signal.generate_flmn(rng, L, N, 0, reality), device="cuda")
    kw = dict(sampling=sampling, reality=reality)
    f = s2b.wigner.inverse(flmn, L, N, **kw)
    ell = np.sqrt((2 * np.arange(L) + 1) / (16 * np.pi**3))[:, None]
    gamma = 2 * np.pi * np.arange(2 * N - 1) / (2 * N - 1)
    ref = 0
    for n in range(-(N - 1), N):
        x = flmn[N - 1 + n] * torch.tensor((-1.0) ** n * ell, device="cuda")
        fn = s2b.inverse(x, L, -n, None, sampling)
        ph = torch.tensor(np.exp(1j * n * gamma), device="cuda")
        ref = ref + ph[:, None, None] * fn
    ref = ref.cpu().numpy()
    assert relerr(f.cpu().numpy(), ref.real if reality else ref) < 1e-10
    g = s2b.wigner.forward(f, L, N, **kw)
    assert relerr(g.cpu().numpy(), flmn.cpu().numpy()) < 1e-10
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fg = s2b.wigner.inverse(flmn, L, N, **kw)
        gg = s2b.wigner.forward(fg, L, N, **kw)
    graph.replay()
    torch.cuda.synchronize()
    assert relerr(fg.cpu().numpy(), f.cpu().numpy()) < 1e-12
    assert relerr(gg.cpu().numpy(), flmn.cpu().numpy()) < 1e-10
