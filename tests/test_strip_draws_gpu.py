"""The strike strip on its own draws: the same Philox blocks in numpy, paths
and payoffs in FP64, at the edges of the kernel's tables and splits: step counts
around the q table's end (256 counter blocks), partial last blocks, partial
warps, one strike (sums per lane) and several, the sample counts where the last
block sums the rows and where a launch does, where few samples spread over the
SMs, and past one resident grid.

Tolerance: a step rounds |y| < 2 by at most 2^-23 and its normal carries about
1e-6 of sigma sqrt(dt); a price is a mean of spots near 100, each off by at most
100 (steps 2^-23 + 2e-5)."""
import math

import numpy as np
import pytest
from scipy.special import ndtri

import openferric_b200 as of
from openferric_b200 import OptionType
from openferric_b200.engines import price_strike_strip
from oracle.book_oracle import _pair, _unif, philox4x32_10

pytestmark = pytest.mark.gpu

TAG, S0, T, MU = 0x53545250, 100.0, 1.0, 0.03
H = dict(kappa=2.0, theta=0.04, xi=0.5, rho=-0.7, v0=0.04)


def _gen(model, steps):
    if model == "gbm":
        return of.GbmPathGenerator(of.Gbm(MU, 0.25), S0, T, steps)
    return of.HestonPathGenerator(of.Heston(MU, **H), S0, T, steps, "qe" if model == "qe" else "euler")


def _paths(model, steps, samples, seed, sign):
    """Terminal spots of the samples (sign -1: their antithetic twins)."""
    lo, dt = np.arange(samples, dtype=np.uint64), T / steps
    y, v = np.zeros(samples), np.full(samples, H["v0"])
    spb = 4 if model == "gbm" else 2
    for b in range(0, steps, spb):
        r = philox4x32_10(np.full_like(lo, b // spb), lo, np.zeros_like(lo), np.full_like(lo, TAG), seed)
        if model == "gbm":
            for z in (_pair(r[0], r[1]) + _pair(r[2], r[3]))[:steps - b]:
                y += (MU - 0.5 * 0.25 ** 2) * dt + 0.25 * math.sqrt(dt) * sign * z
            continue
        for k in range(min(2, steps - b)):
            if model == "heston":
                z1, z2 = (sign * z for z in _pair(r[2 * k], r[2 * k + 1]))
                sv = np.sqrt(v * dt)
                y += (MU - 0.5 * v) * dt + sv * (H["rho"] * z1 + math.sqrt(1 - H["rho"] ** 2) * z2)
                v = np.maximum(v + H["kappa"] * (H["theta"] - v) * dt + H["xi"] * sv * z1, 0.0)
                continue
            u, zx = _unif(r[2 * k]), sign * ndtri(_unif(r[2 * k + 1]))
            u = u if sign > 0 else 1.0 - u
            e = math.exp(-H["kappa"] * dt)
            x2 = H["xi"] ** 2
            m = H["theta"] + (v - H["theta"]) * e
            psi = (v * x2 * e * (1 - e) / H["kappa"] + H["theta"] * x2 * (1 - e) ** 2 / (2 * H["kappa"])) / m ** 2
            t = 2.0 / psi
            with np.errstate(invalid="ignore", divide="ignore"):
                b2 = t - 1 + np.sqrt(np.maximum(t * (t - 1), 0))
                vq = m / (1 + b2) * (np.sqrt(np.maximum(b2, 0)) + ndtri(u)) ** 2
                p = (psi - 1) / (psi + 1)
                ve = np.where(u <= p, 0.0, np.log((1 - p) / (1 - u)) * m / (1 - p))
            vn = np.where(psi <= 1.5, vq, ve)
            kr = H["kappa"] * H["rho"] / H["xi"] - 0.5
            y += MU * dt - H["rho"] * H["kappa"] * H["theta"] * dt / H["xi"] + (0.5 * dt * kr - H["rho"] / H["xi"]) * v \
                + (0.5 * dt * kr + H["rho"] / H["xi"]) * vn + np.sqrt(0.5 * dt * (1 - H["rho"] ** 2) * (v + vn)) * zx
            v = vn
    return S0 * np.exp(y)


@pytest.mark.parametrize("model,steps,samples,anti,strikes", [
    ("gbm", 1, 1, False, 1), ("gbm", 2, 31, True, 1), ("gbm", 3, 33, False, 2), ("gbm", 6, 4737, False, 1),
    ("gbm", 1024, 257, False, 41), ("gbm", 1027, 65, True, 33), ("gbm", 5, 303_105, False, 1),
    ("gbm", 2, 303_103, True, 3),
    ("heston", 1, 33, False, 1), ("heston", 512, 65, True, 3), ("heston", 515, 1025, False, 64),
    ("heston", 4, 303_105, False, 41), ("heston", 3, 20_000, False, 128), ("qe", 5, 2049, True, 1),
    ("qe", 515, 65, False, 5)])
@pytest.mark.parametrize("tile", [0, 1, 2])
def test_strip_prices_its_own_draws(model, steps, samples, anti, strikes, tile):
    ks = np.linspace(85.0, 115.0, strikes)
    got = price_strike_strip(_gen(model, steps), OptionType.Call, ks, 2 * samples if anti else samples, 9, 1.0,
                             antithetic=anti, tile_ilp=tile)
    ends = [_paths(model, steps, samples, 9, s) for s in ((1, -1) if anti else (1,))]
    tol = S0 * (steps * 2.0 ** -23 + 2e-5)
    for k, (p, se) in zip(ks, got):
        x = sum(np.maximum(s - k, 0.0) for s in ends) / len(ends)
        assert abs(p - x.mean()) <= tol, (k, p, x.mean())
        if samples > 1:
            assert abs(se - x.std(ddof=1) / math.sqrt(samples)) <= tol / math.sqrt(samples)
