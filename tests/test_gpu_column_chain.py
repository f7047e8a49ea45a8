"""The MW / MWSS column chain at the band-limits where its transforms change: the shared-memory
passes up to L = 191, the register engine from there on, 4L a power of two, 6L - 1 against the
powers of two, and the largest working lengths with the first band-limit beyond."""

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
@pytest.mark.parametrize("L", [2, 3, 16, 64, 85, 128, 191, 192, 193, 256])
@pytest.mark.parametrize("spin,reality", [(0, False), (1, False), (0, True)])
def test_forward_against_oracle(s2b, rng, sampling, L, spin, reality):
    """White noise on the grid: both parities, the self-mirrored samples and the Nyquist bin
    count (tolerances: the float64 path's and float32 path's bounds on the whole transform)."""
    shape = s2b.spherical.f_shape(L, sampling)
    f = rng.standard_normal(shape) + (0 if reality else 1j * rng.standard_normal(shape))
    ref = oracle.spherical.forward(f, L, spin, None, sampling, reality=reality, backend="c")
    for precision, tol in (("f64", 1e-10), ("f32", 1e-5)):
        y = s2b.forward(f, L, spin, None, sampling, reality=reality, precision=precision)
        assert relerr(y, ref) < tol, (precision, relerr(y, ref))


@pytest.mark.parametrize("sampling", ["mw", "mwss"])
@pytest.mark.parametrize("precision,L", [("f64", 341), ("f64", 342), ("f64", 682), ("f64", 683),
                                         ("f32", 682), ("f32", 683), ("f32", 1365),
                                         ("f32", 1366)])
def test_round_trip_at_the_length_limits(s2b, rng, sampling, precision, L):
    flm = oracle.signal.generate_flm(rng, L, 0, 0, False)
    f = s2b.inverse(flm, L, 0, None, sampling, precision=precision)
    y = s2b.forward(f, L, 0, None, sampling, precision=precision)
    assert relerr(y, flm) < (1e-10 if precision == "f64" else 1e-5), relerr(y, flm)


@pytest.mark.parametrize("L", [64, 128])
def test_short_power_of_two_error(s2b, L):
    """MW float at the powers of two below 192 runs the shared-memory passes. With every twiddle
    from the table the error over five maps of noise is 3.3e-7 (L = 64) and 3.6e-7 (L = 128), with
    twiddles squared in float 4.1e-7 and 4.2e-7; run to run it varies by 1e-9."""
    rng = np.random.default_rng(5)
    e = []
    for _ in range(5):
        f = (rng.standard_normal((L, 2 * L - 1)) + 1j * rng.standard_normal((L, 2 * L - 1)))
        f = f.astype(np.complex64)
        ref = oracle.spherical.forward(f.astype(complex), L, 0, None, "mw", backend="c")
        y = s2b.forward(f, L, precision="f32")
        e.append(np.linalg.norm(y - ref) / np.linalg.norm(ref))
    assert np.mean(e) < 3.85e-7, e


@pytest.mark.parametrize("sampling", ["mw", "mwss"])
@pytest.mark.parametrize("L", [341, 342, 682, 683])
@pytest.mark.parametrize("spin,reality", [(0, True), (1, False)])
def test_noise_at_the_length_limits(s2b, rng, sampling, L, spin, reality):
    """White noise at the working lengths' limits (6L - 1 against 2048 and 4096, in double 4096 the
    last): odd columns' own samples and the Nyquist bin count here, a round trip sees neither."""
    shape = s2b.spherical.f_shape(L, sampling)
    f = rng.standard_normal(shape) + (0 if reality else 1j * rng.standard_normal(shape))
    ref = oracle.spherical.forward(f, L, spin, None, sampling, reality=reality, backend="c")
    for precision, tol in (("f64", 1e-10), ("f32", 1e-5)):
        y = s2b.forward(f, L, spin, None, sampling, reality=reality, precision=precision)
        assert relerr(y, ref) < tol, (precision, relerr(y, ref))


@pytest.mark.parametrize("sampling,L", [("mw", 1365), ("mwss", 1366)])
def test_noise_at_the_longest_length(s2b, rng, sampling, L):
    """Float: 6L - 1 = 8189 on the engine's 8192 points, and the first band-limit beyond it."""
    shape = s2b.spherical.f_shape(L, sampling)
    f = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    ref = oracle.spherical.forward(f, L, 1, None, sampling, backend="c")
    y = s2b.forward(f, L, 1, None, sampling, precision="f32")
    assert relerr(y, ref) < 1e-5, relerr(y, ref)


@pytest.mark.parametrize("sampling", ["mw", "mwss"])
@pytest.mark.parametrize("L", [150, 192, 200, 256])
@pytest.mark.parametrize("spin,reality", [(0, False), (0, True), (-2, False)])
def test_precompute_forward_against_on_the_fly(s2b, rng, sampling, L, spin, reality):
    """The chain's raw layout (precompute forward) on both routes, on white noise: the same map by
    the on-the-fly transform, whose chain the tests above hold to the oracle."""
    shape = s2b.spherical.f_shape(L, sampling)
    f = rng.standard_normal(shape) + (0 if reality else 1j * rng.standard_normal(shape))
    ref = s2b.forward(f, L, spin, None, sampling, reality=reality)
    for precision, tol in (("f64", 1e-10), ("f32", 1e-5)):
        y = s2b.precompute.forward(f, L, spin, None, sampling, reality, precision=precision)
        assert relerr(y, ref) < tol, (precision, relerr(y, ref))
