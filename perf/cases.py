"""The transforms that are timed: listed cases, drawn ones and their float64 values.

Every case is one pass through the package's public calls, as a program that has its maps or
coefficients on the GPU makes it. The families:

sht         inverse of one set of coefficients and forward of one set of maps
grad        map and gradient of a least-squares loss through the inverse
wigner      SO(3) inverse and forward by the recursion
fw          SO(3) inverse and forward by the Fourier-Wigner planes
precompute  inverse and forward of many maps through a kernel table
uneven      inverse and forward of maps of mixed sizes, spins and samplings (BatchedSHT)
rotate      rotation of coefficients by three Euler angles

The float64 values come from the degree recursion of d^l_{mn} in difference form (plain numpy
and torch, none of the package's code); maps given to the forward transforms are synthesised
with the same recursion, so they depend on the seed alone.
"""

import functools
import math
import random

import numpy as np
import torch

import s2fft_b200

_SPINS = (0, 0, 1, 2, -2, 3)


# ---------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------
def _sht(name, sampling, L, spin, precision, maps=1, nside=0, reality=False, iters=0):
    return dict(name=name, family="sht", sampling=sampling, L=L, spin=spin,
                precision=precision, maps=maps, nside=nside, reality=reality, iters=iters)


def listed():
    return [
        # an interactive call at the default precision, where launches and host time count
        _sht("mw128_f64", "mw", 128, 0, "f64"),
        # an odd band-limit, spin-2 (polarisation) maps, three at a time, with pole rings
        _sht("mwss301_spin2_f64_x3", "mwss", 301, 2, "f64", maps=3),
        # the headline size in both precisions
        _sht("mw1024_f32", "mw", 1024, 0, "f32"),
        _sht("mw1024_f64", "mw", 1024, 0, "f64"),
        # a large polarisation map on a ragged band-limit
        _sht("gl1500_spin2_f32", "gl", 1500, 2, "f32"),
        # a real sky map analysed with three refinement iterations
        _sht("healpix256_real_iter3_f32", "healpix", 512, 0, "f32", nside=256, reality=True,
             iters=3),
        # one optimisation step on the coefficients of a map
        dict(name="grad_mw1024_f32", family="grad", sampling="mw", L=1024, spin=0,
             precision="f32"),
        # directional wavelet sizes on SO(3), by either path
        dict(name="wigner_mw128_n8_f32", family="wigner", sampling="mw", L=128, N=8,
             precision="f32"),
        dict(name="fw_mw256_n8_f64", family="fw", sampling="mw", L=256, N=8, precision="f64"),
        # a stack of polarisation maps through a kept kernel table on the tensor cores
        dict(name="precompute_gl512_spin2_x64_bf16x3", family="precompute", sampling="gl",
             L=512, spin=2, precision="bf16x3", maps=64),
        # a queue of maps of mixed sizes
        dict(name="uneven32_f32", family="uneven", maps=32, Lmin=64, Lmax=512, mix=11,
             precision="f32"),
        # a change of frame for a whole set of coefficients
        dict(name="rotate1024_f64", family="rotate", L=1024, maps=1, precision="f64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["sht"] * 8 + ["grad", "wigner", "fw", "precompute", "uneven", "rotate"])
    precision = rng.choice(["f32", "f64"])
    if family == "sht":
        sampling = rng.choice(["mw", "mwss", "dh", "gl", "healpix"])
        if sampling == "healpix":
            nside = _log_int(rng, 16, 256)
            L = rng.choice([2 * nside, 2 * nside + rng.randrange(1, nside)])
            reality = rng.random() < 0.7
            return dict(family="sht", sampling="healpix", L=L, spin=0, precision=precision,
                        maps=1, nside=nside, reality=reality, iters=rng.choice([0, 1, 3]))
        L = _log_int(rng, 32, 1200)
        spin = rng.choice(_SPINS)
        maps = max(1, min(rng.choice([1, 1, 1, 2, 5, 16]), int((1000 / L) ** 3)))
        reality = spin == 0 and rng.random() < 0.3
        return dict(family="sht", sampling=sampling, L=L, spin=spin, precision=precision,
                    maps=maps, nside=0, reality=reality, iters=0)
    if family == "grad":
        return dict(family="grad", sampling=rng.choice(["mw", "mwss", "gl"]),
                    L=_log_int(rng, 32, 1024), spin=rng.choice(_SPINS), precision=precision)
    if family == "wigner":
        return dict(family="wigner", sampling=rng.choice(["mw", "mwss", "gl"]),
                    L=_log_int(rng, 32, 256), N=rng.randrange(2, 9), precision=precision)
    if family == "fw":
        return dict(family="fw", sampling=rng.choice(["mw", "mwss"]),
                    L=_log_int(rng, 32, 256), N=rng.randrange(2, 9), precision=precision)
    if family == "precompute":
        L = _log_int(rng, 32, 400)
        return dict(family="precompute", sampling=rng.choice(["gl", "dh", "mw"]), L=L,
                    spin=rng.choice(_SPINS), precision=rng.choice(["f32", "bf16x3"]),
                    maps=_log_int(rng, 1, 64))
    if family == "uneven":
        return dict(family="uneven", maps=rng.randrange(8, 33), Lmin=64,
                    Lmax=rng.choice([128, 256, 512]), mix=rng.randrange(1 << 16),
                    precision="f32")
    return dict(family="rotate", L=_log_int(rng, 64, 1024), maps=rng.choice([1, 1, 2]),
                precision=precision)


def _specs(case):
    """(L, spin, sampling) of every map of an uneven case."""
    rng = random.Random(case["mix"])
    sizes = [s for s in (64, 128, 256, 512) if case["Lmin"] <= s <= case["Lmax"]]
    return [(rng.choice(sizes), rng.randrange(4), rng.choice(["mw", "mwss", "dh", "gl"]))
            for _ in range(case["maps"])]


# ---------------------------------------------------------------------------------------
# grids
# ---------------------------------------------------------------------------------------
def _ntheta(L, sampling, nside=0):
    return {"mw": L, "mwss": L + 1, "gl": L, "dh": 2 * L, "healpix": 4 * nside - 1}[sampling]


def _nphi(L, sampling):
    return 2 * L if sampling == "mwss" else 2 * L - 1


@functools.lru_cache(maxsize=16)
def _gauss(L):
    """Gauss-Legendre colatitudes in increasing order and weights, in long double: numpy's
    nodes after one Newton step."""
    x = np.polynomial.legendre.leggauss(L)[0][::-1].astype(np.longdouble)

    def legendre(x):
        p0, p1 = np.ones_like(x), x.copy()
        for l in range(1, L):
            p0, p1 = p1, ((2 * l + 1) * x * p1 - l * p0) / (l + 1)
        return p0, p1

    if L == 1:
        return np.array([np.pi / 2]).astype(np.longdouble), np.array([2.0])
    pm, p = legendre(x)
    dp = L * (x * p - pm) / (x * x - 1)
    x = x - p / dp
    pm, p = legendre(x)
    dp = L * (x * p - pm) / (x * x - 1)
    return np.arccos(x), (2 / ((1 - x * x) * dp * dp)).astype(np.float64)


_PI = np.longdouble("3.14159265358979323846264338327950288")


def _thetas(L, sampling, nside=0):
    if sampling == "gl":
        return _gauss(L)[0]
    t = np.arange(_ntheta(L, sampling, nside)).astype(np.longdouble)
    if sampling == "mw":
        return (2 * t + 1) * _PI / (2 * L - 1)
    if sampling == "mwss":
        return t * _PI / L
    if sampling == "dh":
        return (2 * t + 1) * _PI / (4 * L)
    r = t + 1  # HEALPix: 1 - |z| is (r / nside)^2 / 3 in the caps
    r = np.minimum(r, 4 * nside - r)
    y = np.where(r < nside, r * r / (3 * np.longdouble(nside) ** 2),
                 2 * r / (3 * np.longdouble(nside)) - np.longdouble(1) / 3)
    half = 2 * np.arcsin(np.sqrt(y / 2))
    return np.where(t < 2 * nside, half, _PI - half)


def _ring_weights(L, sampling, nside=0):
    """Weights of the theta sum that makes the integral over sin(theta) d theta."""
    if sampling == "gl":
        return _gauss(L)[1]
    th = _thetas(L, sampling, nside).astype(np.float64)
    if sampling == "dh":
        k = 2 * np.arange(L) + 1
        return 2 / L * np.sin(th) * (np.sin(np.outer(th, k)) / k).sum(axis=1)
    return None


def _hp_lengths(nside):
    r = np.arange(1, 4 * nside)
    return 4 * np.minimum(np.minimum(r, 4 * nside - r), nside)


def _hp_phi0(nside):
    r = np.arange(1, 4 * nside)
    n = _hp_lengths(nside)
    belt = (r >= nside) & (r <= 3 * nside)
    return np.where(belt, ((r - nside + 1) % 2) * np.pi / n, np.pi / n)


# ---------------------------------------------------------------------------------------
# d^l_{mn} in float64
# ---------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _seeds(m, n, beta, precise):
    """d^{l0}_{mn}(beta) [beta, column] at l0 = max(|m|, |n|), in closed form."""
    real = np.longdouble if precise else np.float64
    l0 = np.maximum(np.abs(m), np.abs(n))
    sign = np.where((m - n) % 2, -1.0, 1.0)
    a, b = m >= np.abs(n), -m >= np.abs(n)
    c, d = n >= np.abs(m), -n >= np.abs(m)
    k = np.select([a, b, c, d], [n, -n, m, -m])
    sign = np.select([a, b, c, d], [sign, np.ones_like(sign), np.ones_like(sign), sign])
    lf = np.concatenate([[0], np.cumsum(np.log(np.arange(1, 2 * l0.max() + 1).astype(
        np.longdouble)))]).astype(real)
    binom = (lf[2 * l0] - lf[l0 + k] - lf[l0 - k]) / 2
    half = beta.astype(np.longdouble) / 2
    logc, logs = np.log(np.cos(half)).astype(real), np.log(np.sin(half)).astype(real)
    if precise:
        e = binom + (l0 + k) * logc[:, None] + (l0 - k) * logs[:, None]
        return torch.from_numpy((sign * np.exp(e)).astype(np.float64)).to(_device())

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).to(_device())

    e = dev(binom) + dev(l0 + k) * dev(logc)[:, None] + dev(l0 - k) * dev(logs)[:, None]
    return dev(sign) * torch.exp(e)


@functools.lru_cache(maxsize=4)
def _precise_table(L, M, n):
    """Long double A_l(m, n) and 1 - B_l - A_l - A_{l+1} for |m| < M, l <= L, as float64."""
    l = np.arange(L + 1).astype(np.longdouble)[:, None]
    m = np.arange(-(M - 1), M).astype(np.longdouble)[None, :]
    with np.errstate(divide="ignore", invalid="ignore"):
        A = np.sqrt(np.maximum(l * l - m * m, 0) * np.maximum(l * l - n * n, 0)
                    / (l * l * (4 * l * l - 1)))
        B = m * n / (l * (l + 1))
    A[0], B[0] = 0, 0
    gap = 1 - B[:-1] - A[:-1] - A[1:]
    return A.astype(np.float64), gap.astype(np.float64)


def _wigner_rows(L, m, n, beta, precise=False, table=None):
    """Yields (l, D) with D[beta, column] = sqrt((2l + 1) / 2) d^l_{mn}(beta), 0 < beta <= pi/2:
    D_{l+1} - D_l = A_l/A_{l+1} (D_l - D_{l-1}) + (gap_l - (1 - cos beta))/A_{l+1} D_l."""
    dev = _device()
    l0 = np.maximum(np.abs(m), np.abs(n))
    seed = _seeds(m, n, beta, precise)
    y = torch.from_numpy((2 * np.sin(beta.astype(np.longdouble) / 2) ** 2).astype(
        np.float64)).to(dev)[:, None]
    l0t = torch.from_numpy(l0).to(dev)
    mt, nt = (torch.from_numpy(v.astype(np.float64)).to(dev) for v in (m, n))

    def coef(l):
        if table is not None:
            return table[0][l], table[1][l] if l < L else None
        if l == 0:
            return torch.zeros_like(mt), None
        q = (l * l - mt * mt).clamp(min=0) * (l * l - nt * nt).clamp(min=0)
        return torch.sqrt(q) / (l * math.sqrt(4.0 * l * l - 1)), None

    if table is not None:
        table = [torch.from_numpy(t).to(dev) for t in table]
    D = torch.zeros_like(seed)
    diff = torch.zeros_like(seed)
    A, gap = coef(0)
    for l in range(L):
        D = torch.where(l0t == l, seed * math.sqrt(l + 0.5), D)
        yield l, D
        A1, gap1 = coef(l + 1)
        if table is None:
            B = mt * nt / (l * (l + 1)) if l else torch.zeros_like(mt)
            gap = 1 - B - A - A1
        inv = torch.where(l0t <= l, 1 / A1, torch.zeros_like(A1))
        # below its first degree a column stays zero; at it A_l = 0 drops D_{l-1}
        diff = (A * inv) * diff + ((gap - y) * inv) * D
        D = D + diff
        A, gap = A1, gap1


def _blocks(L, spin, theta, precise):
    """Northern and southern rings, with the recursion that serves them:
    d^l_{mn}(pi - beta) = (-1)^{l+m} d^l_{m,-n}(beta). A pole is the limit beta -> 0."""
    north = theta <= _PI / 2
    m = np.arange(-(L - 1), L)
    for south in (False, True):
        rows = np.where(north != south)[0]
        if len(rows):
            n = spin if south else -spin
            beta = np.maximum(_PI - theta[rows] if south else theta[rows],
                              np.longdouble(1e-200))
            table = _precise_table(L, L, n) if precise else None
            yield rows, south, _wigner_rows(L, m, np.full_like(m, n), beta, precise, table)


def _chunks(L, rows, south, it, chunk=16):
    """Stacks of d^l sqrt((2l+1)/4pi) [degree, ring, order] over a few degrees at a time."""
    m = torch.arange(-(L - 1), L, device=_device())
    buf, ls = [], []
    for l, D in it:
        if south:
            D = D * (1 - 2 * ((m + l) % 2)).to(D.dtype)
        buf.append(D / math.sqrt(2 * math.pi))
        ls.append(l)
        if len(ls) == chunk or l == L - 1:
            yield ls[0], ls[-1] + 1, torch.stack(buf)
            buf, ls = [], []


def _synthesis(flm, L, spin, theta, precise=False):
    """Ring spectra [map, ring, 2L-1] of flm [map, L, 2L-1]."""
    flm = flm.to(device=_device(), dtype=torch.complex128)
    out = torch.zeros((flm.shape[0], len(theta), 2 * L - 1), dtype=torch.complex128,
                      device=flm.device)
    parts = torch.view_as_real(flm)  # [map, l, m, 2]
    for rows, south, it in _blocks(L, spin, theta, precise):
        acc = 0
        for la, lb, D in _chunks(L, rows, south, it):
            acc = acc + torch.einsum("crm,bcmz->brmz", D, parts[:, la:lb])
        out[:, torch.from_numpy(rows).to(out.device)] = torch.view_as_complex(acc.contiguous())
    return out * (-1) ** spin


def _analysis(G, L, spin, theta, precise=False):
    """sum over rings of d^l sqrt((2l+1)/4pi) G[map, ring, 2L-1] -> [map, L, 2L-1]."""
    out = torch.zeros((G.shape[0], L, 2 * L - 1), dtype=torch.complex128, device=G.device)
    for rows, south, it in _blocks(L, spin, theta, precise):
        parts = torch.view_as_real(G[:, torch.from_numpy(rows).to(G.device)].contiguous())
        for la, lb, D in _chunks(L, rows, south, it):
            out[:, la:lb] += torch.view_as_complex(
                torch.einsum("crm,brmz->bcmz", D, parts).contiguous())
    return out * (-1) ** spin


# ---------------------------------------------------------------------------------------
# whole transforms in float64
# ---------------------------------------------------------------------------------------
def _map_of(F, L, sampling, nside):
    """Maps of the ring spectra F [map, ring, 2L-1]."""
    if sampling != "healpix":
        n = _nphi(L, sampling)
        pad = torch.zeros(F.shape[:2] + (n,), dtype=F.dtype, device=F.device)
        pad[..., :L] = F[..., L - 1:]
        if L > 1:
            pad[..., n - (L - 1):] = F[..., : L - 1]
        return torch.fft.ifft(pad, norm="forward")
    m = torch.arange(-(L - 1), L, device=F.device)
    F = F * torch.exp(1j * m * torch.from_numpy(_hp_phi0(nside)).to(F.device)[:, None])
    lens = _hp_lengths(nside)
    off = np.concatenate([[0], np.cumsum(lens)])
    out = torch.empty((F.shape[0], off[-1]), dtype=F.dtype, device=F.device)
    for n in np.unique(lens):
        rings = np.where(lens == n)[0]
        bins = torch.zeros((F.shape[0], len(rings), int(n)), dtype=F.dtype, device=F.device)
        bins.index_add_(2, m % int(n), F[:, torch.from_numpy(rings).to(F.device)])
        v = torch.fft.ifft(bins, norm="forward")
        for j, r in enumerate(rings):
            if n < 4 * nside:
                out[:, off[r]:off[r + 1]] = v[:, j]
        if n == 4 * nside:
            out[:, off[rings[0]]:off[rings[-1] + 1]] = v.reshape(F.shape[0], -1)
    return out


def _spectra_of(f, L, sampling, nside):
    """sum_p f exp(-i m phi_p), |m| < L, of every ring."""
    if sampling != "healpix":
        n = _nphi(L, sampling)
        X = torch.fft.fft(f)
        return torch.cat([X[..., n - (L - 1):], X[..., :L]], dim=-1) if L > 1 else X[..., :1]
    lens = _hp_lengths(nside)
    off = np.concatenate([[0], np.cumsum(lens)])
    m = torch.arange(-(L - 1), L, device=f.device)
    out = torch.empty((f.shape[0], len(lens), 2 * L - 1), dtype=torch.complex128,
                      device=f.device)
    for n in np.unique(lens):
        rings = np.where(lens == n)[0]
        v = torch.stack([f[:, off[r]:off[r + 1]] for r in rings], dim=1)
        out[:, torch.from_numpy(rings).to(f.device)] = torch.fft.fft(v)[..., m % int(n)]
    return out * torch.exp(-1j * m * torch.from_numpy(_hp_phi0(nside)).to(f.device)[:, None])


def _inverse64(flm, L, spin, sampling, nside=0, precise=False):
    F = _synthesis(flm, L, spin, _thetas(L, sampling, nside), precise)
    return _map_of(F, L, sampling, nside)


def _forward64(f, L, spin, sampling, nside=0, precise=False):
    f = f.to(device=_device(), dtype=torch.complex128)
    X = _spectra_of(f, L, sampling, nside)
    if sampling in ("dh", "gl"):
        w = torch.from_numpy(_ring_weights(L, sampling)).to(f.device)[:, None]
        return _analysis(X * w * (2 * math.pi / _nphi(L, sampling)), L, spin,
                         _thetas(L, sampling), precise)
    if sampling == "healpix":
        return _analysis(X * (math.pi / (3 * nside * nside)), L, spin,
                         _thetas(L, sampling, nside), precise)
    # MW, MWSS: the rings continue over the circle with the sign (-1)^{m+s}; the trigonometric
    # polynomial through them is evaluated on Gauss-Legendre rings, where the sum is exact
    m = torch.arange(-(L - 1), L, device=f.device)
    par = (1 - 2 * ((m + spin) % 2)).to(torch.float64)
    th = torch.from_numpy(_thetas(L, sampling).astype(np.float64)).to(f.device)
    if sampling == "mw":
        C = torch.cat([X, (X[:, : L - 1] * par).flip(1)], dim=1)
        th = torch.cat([th, 2 * math.pi - th[: L - 1].flip(0)])
    else:
        C = torch.cat([X, (X[:, 1:L] * par).flip(1)], dim=1)
        th = torch.cat([th, 2 * math.pi - th[1:L].flip(0)])
    g = torch.from_numpy(_gauss(L)[0].astype(np.float64)).to(f.device)
    E = torch.exp(1j * torch.outer(m.to(torch.float64), th))  # [k, theta]
    coef = torch.einsum("kt,btm->bkm", E.conj(), C) / len(th)
    G = torch.einsum("kg,bkm->bgm", torch.exp(1j * torch.outer(m.to(torch.float64), g)), coef)
    w = torch.from_numpy(_gauss(L)[1]).to(f.device)[:, None]
    return _analysis(G * w * (2 * math.pi / _nphi(L, sampling)), L, spin, _gauss(L)[0], precise)


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _rdtype(case):
    return torch.float64 if case["precision"] == "f64" else torch.float32


def _cdtype(case):
    return torch.complex128 if case["precision"] == "f64" else torch.complex64


def _random_flm(gen, count, L, spin, reality=False):
    """N(0,1) coefficients, zero outside |m| <= l and below |spin| [count, L, 2L-1]."""
    x = torch.view_as_complex(torch.randn((count, L, 2 * L - 1, 2), generator=gen,
                                          dtype=torch.float64, device=_device()))
    l = torch.arange(L, device=x.device)[:, None]
    m = torch.arange(-(L - 1), L, device=x.device)[None, :]
    x = x * ((m.abs() <= l) & (l >= abs(spin)))
    if reality:
        sgn = (1 - 2 * (m % 2)).to(torch.float64)
        x = torch.where(m < 0, sgn * x.flip(-1).conj(), x)
        x = torch.where(m == 0, x.real.to(x.dtype), x)
    return x


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(seed)


def _sht_inputs(case, seed):
    L, spin, real = case["L"], case["spin"], case.get("reality", False)
    gen = _generator(seed)
    a = _random_flm(gen, case["maps"], L, spin, real).to(_cdtype(case))
    b = _random_flm(gen, case["maps"], L, spin, real)
    f = _inverse64(b, L, spin, case["sampling"], case.get("nside", 0))
    f = f.real.to(_rdtype(case)) if real else f.to(_cdtype(case))
    return a, f.contiguous()


def _grad_inputs(case, seed):
    L, spin = case["L"], case["spin"]
    gen = _generator(seed)
    flm = _random_flm(gen, 1, L, spin)[0].to(_cdtype(case))
    shape = (_ntheta(L, case["sampling"]), _nphi(L, case["sampling"]), 2)
    g = torch.view_as_complex(torch.randn(shape, generator=gen, dtype=torch.float64,
                                          device=_device()))
    return flm, g.to(_cdtype(case))


def _so3_coefficients(case, gen):
    L, N = case["L"], case["N"]
    x = torch.cat([_random_flm(gen, 1, L, n) for n in range(-(N - 1), N)])
    return x


def _so3_inverse64(flmn, L, N, sampling, precise=False):
    l = torch.arange(L, device=flmn.device, dtype=torch.float64)
    scale = torch.sqrt((2 * l + 1) / (16 * math.pi ** 3))[:, None]
    fs = [_inverse64((flmn[N - 1 + n] * scale * (-1) ** n)[None], L, -n, sampling,
                     precise=precise)[0] for n in range(-(N - 1), N)]
    return torch.einsum("nk,ntp->ktp", _gamma(N, flmn.device), torch.stack(fs))


def _so3_forward64(f, L, N, sampling, precise=False):
    G = 2 * N - 1
    l = torch.arange(L, device=f.device, dtype=torch.float64)
    scale = torch.sqrt(4 * math.pi / (2 * l + 1))[:, None] * (2 * math.pi / G)
    fn = torch.einsum("nk,ktp->ntp", _gamma(N, f.device).conj(), f)
    return torch.stack([_forward64(fn[N - 1 + n][None], L, -n, sampling,
                                   precise=precise)[0] * scale * (-1) ** n
                        for n in range(-(N - 1), N)])


def _gamma(N, device):
    n = torch.arange(-(N - 1), N, device=device, dtype=torch.float64)
    k = torch.arange(2 * N - 1, device=device, dtype=torch.float64)
    return torch.exp(2j * math.pi * torch.outer(n, k) / (2 * N - 1))


def _so3_inputs(case, seed):
    gen = _generator(seed)
    a = _so3_coefficients(case, gen).to(_cdtype(case))
    f = _so3_inverse64(_so3_coefficients(case, gen), case["L"], case["N"], case["sampling"])
    return a, f.to(_cdtype(case)).contiguous()


def _uneven_inputs(case, seed):
    gen = _generator(seed)
    return [_random_flm(gen, 1, L, spin)[0].to(torch.complex64) for L, spin, _ in _specs(case)]


def _rotate_inputs(case, seed):
    gen = _generator(seed)
    ang = torch.rand(3, generator=gen, dtype=torch.float64, device=_device()).tolist()
    angles = (2 * math.pi * ang[0], 0.1 + 2.9 * ang[1], 2 * math.pi * ang[2])
    return _random_flm(gen, case["maps"], case["L"], 0).to(_cdtype(case)), angles


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def prepare(case, seed):
    family = case["family"]
    state = dict(case=case)
    if family == "sht":
        state["flm"], state["f"] = _sht_inputs(case, seed)
    elif family == "grad":
        flm, state["g"] = _grad_inputs(case, seed)
        state["flm"] = flm.requires_grad_(True)
    elif family in ("wigner", "fw"):
        state["flmn"], state["f"] = _so3_inputs(case, seed)
        if family == "fw":
            state["planes"] = s2fft_b200.fourier_wigner.fourier_wigner_kernel(case["L"])
    elif family == "precompute":
        state["flm"], state["f"] = _sht_inputs(case, seed)
        state["kernels"] = [s2fft_b200.precompute.spin_spherical_kernel(
            case["L"], case["spin"], False, case["sampling"], forward=fwd,
            precision=case["precision"]) for fwd in (False, True)]
    elif family == "uneven":
        state["flms"] = _uneven_inputs(case, seed)
        state["batch"] = s2fft_b200.batch.BatchedSHT(_specs(case), precision="f32")
    else:
        state["flm"], state["angles"] = _rotate_inputs(case, seed)
    return state


def run(state):
    case = state["case"]
    family, L, prec = case["family"], case.get("L"), case["precision"]
    if family == "sht":
        kw = dict(nside=case["nside"] or None, sampling=case["sampling"],
                  reality=case["reality"], precision=prec)
        return dict(f=s2fft_b200.inverse(state["flm"], L, case["spin"], **kw),
                    flm=s2fft_b200.forward(state["f"], L, case["spin"], iter=case["iters"],
                                           **kw))
    if family == "grad":
        f = s2fft_b200.inverse(state["flm"], L, case["spin"], sampling=case["sampling"],
                               precision=prec)
        r = f - state["g"]
        loss = (r.real.square() + r.imag.square()).sum()
        grad, = torch.autograd.grad(loss, state["flm"])
        return dict(f=f.detach(), grad=grad)
    if family == "wigner":
        kw = dict(sampling=case["sampling"], precision=prec)
        return dict(f=s2fft_b200.wigner.inverse(state["flmn"], L, case["N"], **kw),
                    flmn=s2fft_b200.wigner.forward(state["f"], L, case["N"], **kw))
    if family == "fw":
        fw = s2fft_b200.fourier_wigner
        kw = dict(precomps=state["planes"], sampling=case["sampling"], precision=prec)
        return dict(f=fw.inverse_transform(state["flmn"], L, case["N"], **kw),
                    flmn=fw.forward_transform(state["f"], L, case["N"], **kw))
    if family == "precompute":
        pre = s2fft_b200.precompute
        kw = dict(sampling=case["sampling"], precision=prec)
        return dict(f=pre.inverse(state["flm"], L, case["spin"], state["kernels"][0], **kw),
                    flm=pre.forward(state["f"], L, case["spin"], state["kernels"][1], **kw))
    if family == "uneven":
        b = state["batch"]
        b.load(state["flms"])
        b.run()
        return dict(f=[b.maps(i) for i in range(case["maps"])],
                    flm=[b.coefficients(i) for i in range(case["maps"])])
    return s2fft_b200.rotation.rotate_flms(state["flm"], L, state["angles"])


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _sht_work(L, spin, sampling, nside, maps, elem, real=False, passes=2, refine=0):
    """Bytes: coefficients and map once per direction. Flops: for every degree and order one
    recurrence step (4) per mirrored pair of rings and 4 per ring and complex product; ring
    DFTs at 5 n log2 n."""
    nth = _ntheta(L, sampling, nside)
    npix = 12 * nside * nside if sampling == "healpix" else nth * _nphi(L, sampling)
    terms = sum(L - max(m, abs(spin)) for m in range(L))
    if not spin:
        lat = terms * nth * (2 + 4 * (1 if real else 2))
    else:
        lat = terms * nth * (2 * 2 + 4 * 2)
    fft = 5 * npix * math.log2(max(2, npix / nth)) * (0.5 if real else 1)
    per = maps * (elem * (L * (2 * L - 1) + npix * (0.5 if real else 1)))
    n = passes + 2 * refine
    return dict(bytes=int(passes * per), flops=int(n * maps * (lat + fft)))


def work(case):
    family = case["family"]
    elem = 16 if case["precision"] == "f64" else 8
    L = case.get("L")
    if family == "sht":
        return _sht_work(L, case["spin"], case["sampling"], case["nside"], case["maps"], elem,
                         case["reality"], refine=case["iters"])
    if family == "grad":
        return _sht_work(L, case["spin"], case["sampling"], 0, 1, elem)
    if family in ("wigner", "fw"):
        G = 2 * case["N"] - 1
        w = [_sht_work(L, n, case["sampling"], 0, 1, elem) for n in range(G - case["N"] + 1)]
        tot = {k: w[0][k] + 2 * sum(x[k] for x in w[1:]) for k in ("bytes", "flops")}
        return tot
    if family == "precompute":
        kern = 4 * _ntheta(L, case["sampling"]) * L * (2 * L - 1) * (
            2 if case["sampling"] == "mw" else 1)
        w = _sht_work(L, case["spin"], case["sampling"], 0, case["maps"], elem)
        return dict(bytes=w["bytes"] + 2 * kern, flops=w["flops"])
    if family == "uneven":
        w = [_sht_work(Lk, s, sm, 0, 1, elem) for Lk, s, sm in _specs(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    # rotation: L^3 * 2/3 recurrence steps of 4 flops and 8 flops of product for +-m
    steps = sum((L - m) * (L + m) for m in range(L))
    return dict(bytes=2 * elem * case["maps"] * L * (2 * L - 1),
                flops=int(steps * (4 + 16 * case["maps"])))


def tolerance(case):
    """About four times the distance from the float64 values that was measured over the listed
    cases: 4.6e-6 (bf16 triple products), 5.3e-13 (float64) and 9.2e-7 (float32)."""
    if case["family"] == "precompute" and case["precision"] == "bf16x3":
        return {"rel": 2e-5}
    if case["precision"] == "f64":
        return {"rel": 3e-12}
    return {"rel": 4e-6}


# ---------------------------------------------------------------------------------------
# float64 values
# ---------------------------------------------------------------------------------------
def _keep(x, like_real=False):
    return x.real.contiguous() if like_real else x


def _exact_sht(case, seed):
    L, spin, s, nside = case["L"], case["spin"], case["sampling"], case["nside"]
    real = case["reality"]
    flm, f = _sht_inputs(case, seed)
    out = _inverse64(flm, L, spin, s, nside, precise=True)
    f = f.to(torch.complex128)
    y = _forward64(f, L, spin, s, nside, precise=True)
    for _ in range(case["iters"]):
        y = y + _forward64(f - _keep(_inverse64(y, L, spin, s, nside, precise=True), real), L,
                           spin, s, nside, precise=True)
    return dict(f=_keep(out, real), flm=y)


def _exact_grad(case, seed):
    L, spin, s = case["L"], case["spin"], case["sampling"]
    flm, g = _grad_inputs(case, seed)
    f = _inverse64(flm[None], L, spin, s, precise=True)
    X = _spectra_of(f - g.to(torch.complex128)[None], L, s, 0)
    grad = 2 * _analysis(X, L, spin, _thetas(L, s), precise=True)
    return dict(f=f[0], grad=grad[0])


def _exact_rotate(case, seed):
    L = case["L"]
    flm, (alpha, beta, gamma) = _rotate_inputs(case, seed)
    flm = flm.to(torch.complex128)
    orders = np.arange(-(L - 1), L)
    m, n = (v.reshape(-1) for v in np.meshgrid(orders, orders, indexing="ij"))
    flip = beta > math.pi / 2
    b = np.array([_PI - np.longdouble(beta) if flip else np.longdouble(beta)])
    mt = torch.from_numpy(orders.astype(np.float64)).to(flm.device)
    out = torch.zeros_like(flm)
    x = torch.view_as_real(flm * torch.exp(-1j * mt * gamma))
    for l, D in _wigner_rows(L, m, -n if flip else n, b):
        d = D.reshape(2 * L - 1, 2 * L - 1) / math.sqrt(l + 0.5)
        y = torch.einsum("mn,bnz->bmz", d, x[:, l])
        if flip:
            y = y * (1 - 2 * ((mt + l) % 2))[:, None]
        out[:, l] = torch.view_as_complex(y.contiguous()) * torch.exp(-1j * mt * alpha)
    return out


def exact(case, seed):
    family, L = case["family"], case.get("L")
    if family == "sht":
        return _exact_sht(case, seed)
    if family == "grad":
        return _exact_grad(case, seed)
    if family in ("wigner", "fw"):
        flmn, f = _so3_inputs(case, seed)
        args = (L, case["N"], case["sampling"])
        return dict(f=_so3_inverse64(flmn.to(torch.complex128), *args, precise=True),
                    flmn=_so3_forward64(f.to(torch.complex128), *args, precise=True))
    if family == "precompute":
        flm, f = _sht_inputs(case, seed)
        args = (L, case["spin"], case["sampling"])
        return dict(f=_inverse64(flm, *args, precise=True),
                    flm=_forward64(f, *args, precise=True))
    if family == "uneven":
        fs = [_inverse64(x[None], L, spin, s, precise=True)[0]
              for x, (L, spin, s) in zip(_uneven_inputs(case, seed), _specs(case))]
        # the forward runs on the maps of the same pass, so it gives the coefficients back
        return dict(f=fs, flm=[x.to(torch.complex128) for x in _uneven_inputs(case, seed)])
    return _exact_rotate(case, seed)
