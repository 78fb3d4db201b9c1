"""Max-log LLRs over every point with one prior for all (two symbols per step,
by distance) against the oracle, bit for bit: every table size of the chunk
tree, odd counts, unaligned input, one noise value per frame of odd length,
and values at which distances or metrics overflow."""

from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", range(1, 13))
@pytest.mark.parametrize("prior", [0.0, -1.5, None])
def test_tables_against_oracle(k, prior):
    import torch

    from commkit_gb300 import _cuda

    rng = np.random.default_rng(k)
    M = 1 << k
    pts = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(np.complex64)
    logp = rng.uniform(-5, 0, M).astype(np.float32) if prior is None else np.full(M, prior, np.float32)
    labels = rng.permutation(M).astype(np.int32)
    tables = [torch.from_numpy(a).cuda() for a in (pts, logp, labels)]
    launch = _cuda.get_kernel("llr")
    n = 1025
    x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    x[:6] = [np.nan, np.inf, 1e19 + 1j, -1e18, 1e-30j, pts[0]]
    t = torch.from_numpy(x).cuda()
    for s2 in (np.float32(2.5), np.float32(1e20), np.float32(1e-35)):
        for first, count in ((0, n), (0, 1), (1, n - 1), (2, 2), (3, 3)):
            got = launch(t[first : first + count], *tables, k=k, inv_s2=s2, exact=False).cpu().numpy()
            want = oracle.llr_points(x[first : first + count], pts, logp, labels, k, s2, exact=False)
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("family,order", [("psk", 8), ("psk", 16), ("qam", 8), ("qam", 32), ("qam", 128), ("qam", 512)])
def test_frames_against_single_calls(family, order):
    import torch

    import commkit_gb300 as ck

    c = ck.Constellation.psk(order) if family == "psk" else ck.Constellation.qam(order)
    rng = np.random.default_rng(order)
    x = torch.from_numpy((rng.standard_normal((9, 37)) + 1j * rng.standard_normal((9, 37))).astype(np.complex64)).cuda()
    nv = rng.uniform(0.01, 0.5, 9)
    got = ck.compute_llr_frames(x, noise_var=nv, constellation=c, method="maxlog")
    for f in range(9):
        one = ck.compute_llr(x[f].clone(), noise_var=float(nv[f]), constellation=c, method="maxlog")
        np.testing.assert_array_equal(got[f].cpu().numpy(), one.cpu().numpy())


@pytest.mark.parametrize("order", [32, 128, 512])
@pytest.mark.parametrize("form", ["factory", "scaled", "moved", "swapped", "prior"])
def test_cross_qam_against_oracle(order, form):
    """Gray cross QAM by its coordinates, at any scale; a point off the grid,
    two labels exchanged and a prior take the other steps."""
    import torch

    import commkit_gb300 as ck
    from commkit_gb300 import _cuda
    from commkit_gb300.mapping import host_tables

    pts, logp, labels = (a.copy() for a in host_tables(ck.Constellation.qam(order), "points"))
    rng = np.random.default_rng(order)
    if form == "scaled":
        pts = (np.float32(3.7) * pts.real - 1j * np.float32(0.2) * pts.imag).astype(np.complex64)
        pts, labels = pts[::-1].copy(), labels[::-1].copy()
    elif form == "moved":
        pts[order // 3] += np.float32(1e-6)
    elif form == "swapped":
        labels[[1, order - 2]] = labels[[order - 2, 1]]
    elif form == "prior":
        logp[5] = -0.25
    k = int(np.log2(order))
    n = 3001
    x = (pts[rng.integers(0, order, n)] + 0.05 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))).astype(np.complex64)
    x[: n // 3] = rng.choice(pts.real, n // 3) + 1j * rng.choice(pts.imag, n // 3)  # on the grid: ties
    x[n // 3 : n // 2] = 0.5 * (pts[rng.integers(0, order, n // 2 - n // 3)] + pts[0])
    x[-6:] = [np.nan, 1j * np.nan, np.inf, 1e19 + 1j, -1e18, 0]
    tables = [torch.from_numpy(a).cuda() for a in (pts, logp, labels)]
    launch = _cuda.get_kernel("llr")
    for s2 in (np.float32(40.0), np.float32(1e20)):
        got = launch(torch.from_numpy(x).cuda(), *tables, k=k, inv_s2=s2, exact=False).cpu().numpy()
        np.testing.assert_array_equal(got, oracle.llr_points(x, pts, logp, labels, k, s2, exact=False))
