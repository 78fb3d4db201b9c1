"""Exact LLRs of Gray square QAM, uniform and shaped (two symbols per step, base 2)
against a float64 evaluation, where the steps can go wrong: odd counts,
unaligned input, one noise value per frame of odd length, and noise from so
low that half-sums underflow or distances leave the steps' range to so high
that the LLRs vanish."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def exact64(x: np.ndarray, c, s2: np.ndarray) -> tuple[np.ndarray, np.ndarray]:
    """(n, k) float64 LLRs, axis by axis with the axes' log priors as the
    demapper gets them (pmf held at 1e-40 or above, float32), and (n,) largest
    metric magnitudes."""

    def lse(v):
        p = v.max(1, keepdims=True)
        return p[:, 0] + np.log(np.exp(v - p).sum(1))

    llrs = np.zeros((x.size, c.bits_per_symbol))
    most = np.zeros(x.size)
    for axis, coord in zip(c._axes, (x.real, x.imag), strict=True):
        pmf = np.ones(axis.levels.size) if axis.pmf is None else axis.pmf
        logp = np.log(np.clip(pmf, 1e-40, None)).astype(np.float32).astype(np.float64)
        levels = np.asarray(axis.levels).astype(np.float32).astype(np.float64)
        m = logp - (coord.astype(np.float64)[:, None] - levels) ** 2 * s2[:, None]
        most = np.maximum(most, -m.min(1))
        for i, b in enumerate(axis.bits):
            ones = np.asarray(axis.labels)[:, i] != 0
            llrs[:, b] = lse(m[:, ~ones]) - lse(m[:, ones])
    return llrs, most


def check(got, x, c, s2):
    want, most = exact64(x, c, s2)
    # Each of the two metrics rounds its difference (twice, squared), square
    # and scale, and the LLR its difference and factor: 8 half-units of the
    # largest metric; the hardware's 2^x and log2 add 2^-22 each, a few times.
    bound = 2.0**-21 * most[:, None] + 2.0**-19
    err = np.abs(got.reshape(want.shape).astype(np.float64) - want)
    assert np.all(err <= bound), float((err / bound).max())


@pytest.mark.parametrize("order,nu", [(4, None), (16, None), (64, None), (256, None), (16, 0.4), (64, 1.5), (256, 3.0)])
@pytest.mark.parametrize("esn0_db", [-90.0, -20.0, 0.0, 12.0, 19.0, 25.0, 32.0, 45.0, 70.0])
def test_square_qam_against_float64(order, nu, esn0_db):
    import torch

    import commkit_gb300 as ck

    c = ck.Constellation.qam(order)
    if nu is not None:
        c = c.shaped(nu=nu)
    rng = np.random.default_rng(order)
    nv = 10.0 ** (-esn0_db / 10.0)
    n = 2051
    x = rng.choice(np.asarray(c.points), n) + np.sqrt(min(nv, 0.3) / 2) * (
        rng.standard_normal(n) + 1j * rng.standard_normal(n))  # fmt: skip
    x = x.astype(np.complex64)
    s2 = np.full(n, np.float32(1.0 / nv), np.float64)
    t = torch.from_numpy(x).cuda()
    got = ck.compute_llr(t, noise_var=nv, constellation=c, method="exact").cpu().numpy()
    check(got, x, c, s2)
    # An input one symbol into a buffer gives the same bits.
    part = ck.compute_llr(t[1:], noise_var=nv, constellation=c, method="exact").cpu().numpy()
    np.testing.assert_array_equal(part, got[c.bits_per_symbol :])
    one = ck.compute_llr(t[:1], noise_var=nv, constellation=c, method="exact").cpu().numpy()
    np.testing.assert_array_equal(one, got[: c.bits_per_symbol])


@pytest.mark.parametrize("order", [4, 16, 64, 256])
def test_frames_and_nonfinite(order):
    import torch

    import commkit_gb300 as ck
    from commkit_gb300 import compute_llr_frames

    c = ck.Constellation.qam(order)
    rng = np.random.default_rng(1)
    x = (rng.standard_normal((7, 33)) + 1j * rng.standard_normal((7, 33))).astype(np.complex64)
    nv = 10.0 ** (-rng.uniform(0, 30, 7) / 10.0)
    got = compute_llr_frames(torch.from_numpy(x).cuda(), noise_var=nv, constellation=c, method="exact").cpu().numpy()
    check(got, x.reshape(-1), c, np.repeat((1.0 / nv).astype(np.float32), 33).astype(np.float64))
    x = np.array([1e17, np.inf, np.nan, 0.1 + 0.2j, 1j * np.inf, -1e12 + 1j], np.complex64)
    got = ck.compute_llr(torch.from_numpy(x).cuda(), noise_var=0.1, constellation=c, method="exact").cpu().numpy()
    k = c.bits_per_symbol
    got = got.reshape(-1, k)
    assert np.all(np.isfinite(got[[0, 3, 5]]))
    assert np.all(got[0, k // 2] == 0.0)  # on the axis: a tie
    assert np.all(np.isnan(got[[1, 2], : k // 2])) and np.all(np.isnan(got[4, k // 2 :]))


def test_shaped_error_no_larger_than_level_by_level():
    """With priors, the two-symbol steps' error against float64 is, over the
    noise range, no larger than that of the level-by-level method, which the
    same constellation takes with every label bit inverted (the same LLRs,
    negated)."""
    import torch

    import commkit_gb300 as ck

    for order, nu in ((16, 0.5), (16, 1.0), (64, 0.2), (64, 0.5), (64, 1.0), (256, 0.2), (256, 0.5)):
        c = ck.Constellation.qam(order).shaped(nu=nu)
        inverted = ck.Constellation(c.points, 1 - np.asarray(c.bit_labels), c.pmf)
        assert inverted._axes is not None
        rng = np.random.default_rng(order)
        ratios = []
        for esn0_db in range(0, 33, 4):
            nv = 10.0 ** (-esn0_db / 10.0)
            n = 20000
            x = c.points[rng.choice(order, n, p=np.asarray(c.pmf) / np.sum(c.pmf))]
            x = (x + np.sqrt(nv / 2) * (rng.standard_normal(n) + 1j * rng.standard_normal(n))).astype(np.complex64)
            want, _ = exact64(x, c, np.full(n, float(np.float32(1.0 / nv))))
            t = torch.from_numpy(x).cuda()
            got = ck.compute_llr(t, noise_var=nv, constellation=c, method="exact").cpu().numpy()
            levels = -ck.compute_llr(t, noise_var=nv, constellation=inverted, method="exact").cpu().numpy()
            rms = [np.sqrt(np.mean((v.reshape(want.shape).astype(np.float64) - want) ** 2)) for v in (got, levels)]
            ratios.append(rms[0] / rms[1])
        assert np.mean(ratios) <= 1.0, (order, nu, ratios)
