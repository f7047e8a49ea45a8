"""The walk along n behind rotate_flms where it can go wrong: tiles of 64 and 128 orders and
chunks of 128 steps and their neighbours, every fold of beta, angles whose start values lie far
below the double range, and non-finite coefficients."""

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


# a step rounds its factor and its value (a few 1.1e-16) and such errors add up over the at most
# 2L steps of a walk; the oracle's planes carry as much: 2e-13 covers both at these sizes
@pytest.mark.parametrize("L", [2, 63, 64, 65, 128, 129, 130])
@pytest.mark.parametrize("beta", [0.4, np.pi / 2, 2.8, 3.6, -1.0, 9.1])
def test_walk_against_risbo(s2b, rng, L, beta):
    rot = (0.4, beta, -0.9)
    flm = oracle.signal.generate_flm(rng, L, 0, 0, False)
    r = s2b.rotation.rotate_flms(flm, L, rot)
    ref = oracle.rotation.rotate_flms(flm, L, rot)
    assert relerr(r, ref) < 2e-13, relerr(r, ref)


@pytest.mark.parametrize("beta", [0.0, 1e-300, 1e-30, 1e-5, 1e-4, 3e-3, np.pi - 1e-5, np.pi])
def test_walk_near_the_poles(s2b, rng, beta):
    """Start values down to 2^-50000; below sin(beta/2) = 2^-16 the exponents are renewed
    every step."""
    L = 130
    rot = (1.0, beta, 0.3)
    flm = oracle.signal.generate_flm(rng, L, 0, 0, False)
    r = s2b.rotation.rotate_flms(flm, L, rot)
    ref = oracle.rotation.rotate_flms(flm, L, rot)
    assert relerr(r, ref) < 2e-13, relerr(r, ref)


def test_walk_keeps_non_finite_coefficients(s2b, rng):
    """A non-finite coefficient reaches every order of its degree and no other degree."""
    L = 96
    rot = (0.2, 0.7, 0.5)
    flm = oracle.signal.generate_flm(rng, L, 0, 0, False)
    ref = s2b.rotation.rotate_flms(flm, L, rot)
    flm[40, L - 1 + 40] = np.nan
    flm[70, L - 1 - 3] = np.inf
    r = s2b.rotation.rotate_flms(flm, L, rot)
    for l in range(L):
        row = r[l, L - 1 - l:L + l]
        if l in (40, 70):
            assert not np.isfinite(row).any()
        else:
            assert np.array_equal(row, ref[l, L - 1 - l:L + l])
