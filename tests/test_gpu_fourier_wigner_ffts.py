"""The Fourier-Wigner FFT chains where their working lengths and routes change: the shared-memory
passes and, per chain and precision from 256 to 2048 points on, the register engine, power-of-two
rings (mwss) beside Bluestein's, on random SO(3) samples, so that every sampled value counts."""

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


@pytest.mark.parametrize("sampling", ["mw", "mwss"])
@pytest.mark.parametrize("L", [31, 32, 33, 63, 64, 65])
def test_against_oracle(s2b, rng, sampling, L):
    N = 3
    fw = s2b.fourier_wigner
    flmn = oracle.signal.generate_flmn(rng, L, N, 0, False)
    ref = oracle.fourier_wigner.inverse_transform(flmn, L, N, None, False, sampling)
    f = rng.standard_normal(ref.shape) + 1j * rng.standard_normal(ref.shape)
    gref = oracle.fourier_wigner.forward_transform(f, L, N, None, False, sampling)
    for precision, tol in (("f64", 1e-12), ("f32", 1e-5)):
        kw = dict(sampling=sampling, precision=precision)
        assert relerr(fw.inverse_transform(flmn, L, N, **kw), ref) < tol
        assert relerr(fw.forward_transform(f, L, N, **kw), gref) < tol


@pytest.mark.parametrize("sampling,L", [(s, L) for s in ("mw", "mwss") for L in (128, 129, 256)]
                         + [("mwss", 512)])
def test_against_the_recursion(s2b, rng, sampling, L):
    """Larger lengths against the recursion-based transforms of the same library."""
    N = 2
    flmn = oracle.signal.generate_flmn(rng, L, N, 0, False)
    f = s2b.fourier_wigner.inverse_transform(flmn, L, N, sampling=sampling)
    assert relerr(f, s2b.wigner.inverse(flmn, L, N, sampling=sampling)) < 1e-10
    assert relerr(s2b.fourier_wigner.forward_transform(f, L, N, sampling=sampling), flmn) < 1e-10
    kw = dict(sampling=sampling, precision="f32")
    assert relerr(s2b.fourier_wigner.inverse_transform(flmn, L, N, **kw), f) < 1e-5
    assert relerr(s2b.fourier_wigner.forward_transform(f, L, N, **kw), flmn) < 1e-5
