"""Min-sum decoding of codes without circulant structure (rows in 32-row
groups with 16-bit columns, the posterior in shared memory) against the CPU
oracle, bit for bit, at the sizes where the grouping can go wrong."""

from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def staircase_code(ck, N: int, m: int, weight: int, seed: int, punctured: int = 0):
    """Information columns of ``weight`` ones spread evenly over the rows,
    and a staircase parity part."""
    k = N - m
    rng = np.random.default_rng(seed)
    rows = np.concatenate([rng.permutation(m) for _ in range(-(-k * weight // m))])[: k * weight]
    key = np.unique(rows.astype(np.int64) * N + np.repeat(np.arange(k), weight))
    checks = np.concatenate([key // N, np.arange(m), np.arange(1, m)])
    variables = np.concatenate([key % N, k + np.arange(m), k + np.arange(m - 1)])
    return ck.LDPCCode(checks, variables, m, N, punctured)


# N, m, column weight, punctured, frames: layers of a few rows and of one
# row; rows of 4 to 6 (one 16-byte load of columns), 14, 22 and 26 (two to
# four), of many degrees; the largest N of the 16-bit columns and the next;
# variables beyond shared memory in a row's last two edges only, and in more
# (few rows, so that information columns lie there too); punctured parity.
CASES = [
    (24, 12, 2, 0, 3),
    (130, 66, 3, 2, 7),
    (2000, 1000, 3, 0, 40),
    (1999, 777, 3, 5, 700),
    (16200, 4050, 4, 0, 9),
    (12000, 2000, 4, 0, 5),
    (9000, 1000, 3, 0, 5),
    (64800, 32400, 3, 1, 3),
    (64800, 10800, 3, 0, 2),
    (64800, 4000, 1, 0, 2),
    (65535, 30000, 2, 0, 2),
    (65536, 30000, 2, 0, 2),
]


def test_short_batch_in_blocks_that_are_resident():
    """A code of which a block holds two frames and an SM one block: a batch
    of two frames per SM runs as blocks of two."""
    import torch

    import commkit_gb300 as ck

    code = staircase_code(ck, 28500, 14250, 3, seed=4)
    plan = code._plan(0)
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("frame counts of 152 SMs")
    assert plan.workspace_size(301) == plan.workspace_size(302) > plan.workspace_size(300)
    llrs = (1.5 + 2.0 * np.random.default_rng(2).standard_normal((301, code.n))).astype(np.float32)
    row_ptr, cols, _ = code._schedule
    method = ck.MinSum(max_iterations=3)
    r = ck.decode(torch.from_numpy(llrs).cuda(), code=code, method=method)
    want = oracle.decode(llrs, (row_ptr, cols, 28500), k=code.k, scale=method.scale, offset=method.offset,
                         max_iterations=3, early_stop=True)  # fmt: skip
    for g, w in zip((r.bits, r.llrs, r.valid, r.iterations), want, strict=True):
        np.testing.assert_array_equal(g.cpu().numpy().reshape(w.shape), w)


@pytest.mark.parametrize("N,m,weight,punctured,frames", CASES)
@pytest.mark.parametrize("placement", [1, 2])
def test_staircase_codes_equal_oracle(N, m, weight, punctured, frames, placement):
    import torch

    import commkit_gb300 as ck

    code = staircase_code(ck, N, m, weight, seed=N + m, punctured=punctured)
    plan = code._plan(0)
    assert plan.info["quasi_cyclic"] == 0
    rng = np.random.default_rng(7)
    llrs = (2.0 + 2.0 * rng.standard_normal((frames, code.n))).astype(np.float32)
    llrs[0, :8] = [0.0, -0.0, np.inf, -np.inf, 1e30, -1e30, 1e-38, -1e-38]
    x = torch.from_numpy(llrs).cuda()
    row_ptr, cols, _ = code._schedule
    for method in (ck.MinSum(max_iterations=6), ck.MinSum(scale=0.75, offset=0.05, max_iterations=3, early_stop=False)):
        want = oracle.decode(llrs, (row_ptr, cols, N), k=code.k, scale=method.scale, offset=method.offset,
                             max_iterations=method.max_iterations, early_stop=method.early_stop)  # fmt: skip
        for threads in (0, 64, 512 if plan.info["max_row_degree"] > 16 else 1024):
            plan.set_launch(threads, 0, placement)
            r = ck.decode(x, code=code, method=method)
            got = (r.bits.cpu().numpy(), r.llrs.cpu().numpy(), r.valid.cpu().numpy().reshape(-1),
                   r.iterations.cpu().numpy().reshape(-1))  # fmt: skip
            for g, w, what in zip(got, want, ("bits", "llrs", "valid", "iterations"), strict=True):
                np.testing.assert_array_equal(g.reshape(w.shape), w, err_msg=f"{what}, {threads} threads")


@pytest.mark.parametrize("N,m,weight", [(6000, 3000, 3), (3000, 750, 4), (64800, 32400, 3)])
def test_not_a_number_counts_as_absent(N, m, weight):
    """NaN and infinite LLRs, which meet in rows: a NaN magnitude changes no
    minimum, as in the oracle."""
    import torch

    import commkit_gb300 as ck

    code = staircase_code(ck, N, m, weight, seed=N)
    rng = np.random.default_rng(11)
    llrs = (2.0 + 2.0 * rng.standard_normal((3, code.n))).astype(np.float32)
    llrs[0, rng.integers(0, N, 40)] = np.nan
    llrs[1, rng.integers(0, N, 40)] = np.inf
    llrs[1, rng.integers(0, N, 40)] = -np.inf
    llrs[2, N - 3 :] = [np.nan, np.inf, -np.inf]
    row_ptr, cols, _ = code._schedule
    method = ck.MinSum(max_iterations=5)
    r = ck.decode(torch.from_numpy(llrs).cuda(), code=code, method=method)
    want = oracle.decode(llrs, (row_ptr, cols, N), k=code.k, scale=method.scale, offset=method.offset, max_iterations=5,
                         early_stop=True)  # fmt: skip
    for g, w in zip((r.bits, r.llrs, r.valid, r.iterations), want, strict=True):
        np.testing.assert_array_equal(g.cpu().numpy().reshape(w.shape), w)
