"""Small entries of the rotation: with one unit coefficient per degree the rotated coefficients
are single values d^l_{m,n}(beta), known in closed form for n = l, l - 1 and -l, down to the end of
the double range."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def s2b():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import s2fft_b200

    return s2fft_b200


def top_column(L, beta):
    """(sign, log |d^l_{m,l}(beta)|) at [l, L-1+m]:
    d^l_{m,l} = sqrt(binom(2l, l+m)) cos(beta/2)^(l+m) sin(beta/2)^(l-m)."""
    k = np.arange(2 * L).astype(np.longdouble)
    lf = np.concatenate([[0], np.cumsum(np.log(k[1:]))])
    c, s = np.cos(np.longdouble(beta) / 2), np.sin(np.longdouble(beta) / 2)
    l, m = np.arange(L)[:, None], np.arange(-(L - 1), L)[None, :]
    a, b = np.maximum(l + m, 0), np.maximum(l - m, 0)
    e = (lf[2 * l] - lf[np.minimum(a, 2 * L - 1)] - lf[np.minimum(b, 2 * L - 1)]) / 2
    e = e + a * np.log(abs(c)) + b * np.log(abs(s))
    sign = np.where((c < 0) & (a % 2 == 1), -1, 1) * np.where((s < 0) & (b % 2 == 1), -1, 1)
    return np.where(np.abs(m) <= l, sign, 0), e


# a value carries the roundings of the steps from n = l: at most 2L (d_{l,l-1} near beta = 0 comes
# from the walk of order -l), each with a few of 1.1e-16, four say: 1e-15 L
@pytest.mark.parametrize("L,beta", [
    (L, b) for L in (65, 300)
    for b in (1e-6, 1e-4, 0.03, 0.2, 0.8, np.pi / 2, 2.6, 3.1, -0.7, 5.0)] + [(1601, 0.8)])
def test_tiny_entries_keep_their_digits(s2b, L, beta):
    l, m = np.arange(L)[:, None], np.arange(-(L - 1), L)[None, :]
    sign, e = top_column(L, beta)
    # one step along n: sqrt(2l) d_{m,l-1} = 2 (l cos(beta) - m) / sin(beta) d_{m,l}; its error is
    # that of the two terms of l cos(beta) - m, written with the smaller of 1 -+ cos(beta)
    lb = np.longdouble(beta)
    fold = -1 if np.cos(beta) < 0 else 1
    y = 2 * (np.sin(lb / 2) if fold > 0 else np.cos(lb / 2)) ** 2
    unit = 2 / (np.sin(lb) * np.sqrt(np.maximum(2 * l, 1).astype(np.longdouble)))
    step, terms = fold * (l - fold * m - l * y) * unit, (abs(l - fold * m) + l * y) * abs(unit)
    with np.errstate(under="ignore"):
        d = sign * np.exp(e)  # d_{m,l}
    cases = {"l": (np.arange(L), d, abs(d)),
             "l-1": (np.arange(L) - 1, d * step, abs(d) * terms),
             # d_{m,-l} = (-1)^(l+m) d_{-m,l}
             "-l": (-np.arange(L), d[:, ::-1] * np.where((l + m) % 2, -1, 1), abs(d[:, ::-1]))}
    smallest = 1.0
    least = 1e-255  # 2^-881 at L = 300, beta = 1e-4 is the largest of the kernel's limits here
    for name, (n, ref, scale) in cases.items():
        flm = np.zeros((L, 2 * L - 1), complex)
        flm[np.arange(L), L - 1 + n] = 1
        if name == "l-1":
            flm[0] = ref[0] = 0
        r = s2b.rotation.rotate_flms(flm, L, (0.0, beta, 0.0))
        normal = (abs(ref) > least) & (sign != 0)
        smallest = min(smallest, abs(ref[normal]).min())
        err = abs(r - ref)
        assert (err[normal] <= 1e-15 * L * scale[normal]).all(), (name, (err / scale)[normal].max())
        assert (err[~normal] <= 2 * least).all(), name
    assert smallest < 1e-15, smallest


@pytest.mark.parametrize("beta,least", [(1e-12, 1e-290), (1e-40, 1e-260), (-1e-60, 1e-240),
                                        (1e-120, 1e-180), (1e-149, 1e-151)])
def test_tiny_angles(s2b, beta, least):
    """d^l_{m,l} for angles whose step factors reach 2^500: sin(beta/2)^(l-m) down to the limit
    2^(-1021 + bits) of the walk, bits = log2(2 sqrt(2L) cot(beta/2)) rounded up (about `least`)."""
    L = 65
    sign, e = top_column(L, beta)
    with np.errstate(under="ignore"):
        ref = sign * np.exp(e)
    flm = np.zeros((L, 2 * L - 1), complex)
    flm[np.arange(L), L - 1 + np.arange(L)] = 1
    r = s2b.rotation.rotate_flms(flm, L, (0.0, beta, 0.0))
    normal = (abs(ref) > least) & (sign != 0)
    assert np.count_nonzero(normal) >= 2 * L - 1
    err = abs(r - ref)
    assert (err[normal] <= 1e-15 * L * abs(ref[normal])).all(), (err / abs(ref))[normal].max()
    assert (err[~normal] <= 2 * least).all()


@pytest.mark.parametrize("L", [1, 2, 65, 130])
@pytest.mark.parametrize("beta", [0.0, 1e-155, 1e-300])
def test_identity_leaves_zeros(s2b, rng, L, beta):
    """No rotation: zeros stay zeros, and the coefficients themselves to rounding."""
    flm = np.zeros((L, 2 * L - 1), complex)
    flm[np.arange(L), L - 1 + np.arange(L) // 2] = rng.standard_normal(L) + 1j
    r = s2b.rotation.rotate_flms(flm, L, (0.0, beta, 0.0))
    assert (r[flm == 0] == 0).all()
    assert np.abs(r - flm).max() <= 1e-15 * L * np.abs(flm).max()
