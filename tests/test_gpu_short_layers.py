"""Min-sum decoding of codes without circulant structure whose layers are a
few rows each (schedules given through the plan, as the C ABI takes them)
against the CPU oracle, bit for bit, and within the workspace asked for."""

from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def staircase_rows(N: int, m: int, weight: int, seed: int):
    """CSR rows: information columns of ``weight`` ones spread evenly over the
    rows, and a staircase parity part."""
    k = N - m
    rng = np.random.default_rng(seed)
    rows = np.concatenate([rng.permutation(m) for _ in range(-(-k * weight // m))])[: k * weight]
    key = rows.astype(np.int64) * N + np.repeat(np.arange(k), weight)
    j = np.arange(m, dtype=np.int64)
    key = np.unique(np.concatenate([key, j * N + k + j, j[1:] * N + k + j[:-1]]))
    row_ptr = np.zeros(m + 1, np.int32)
    np.cumsum(np.bincount(key // N, minlength=m), out=row_ptr[1:])
    return row_ptr, (key % N).astype(np.int32)


def check_serial(N, m, weight, frames, placement):
    import torch

    import commkit_gb300 as ck
    from commkit_gb300 import _device, _lib
    from commkit_gb300.coding import _Plan, _rule_args

    row_ptr, cols = staircase_rows(N, m, weight, seed=N + m)
    plan = _Plan(row_ptr, cols, np.arange(m + 1, dtype=np.int32), m, N)  # a layer per row
    assert plan.info["quasi_cyclic"] == 0
    plan.set_launch(0, 0, placement)
    k, n = N - m, N - 1  # one punctured bit
    llrs = (2.0 + 2.0 * np.random.default_rng(5).standard_normal((frames, n))).astype(np.float32)
    llrs[0, :8] = [0.0, -0.0, np.inf, -np.inf, 1e30, np.nan, 1e-38, -1e-38]
    x = torch.from_numpy(llrs).cuda()
    out = torch.empty_like(x)
    bits = torch.empty((frames, k), dtype=torch.int8, device="cuda")
    iters = torch.empty(frames, dtype=torch.int32, device="cuda")
    valid = torch.empty(frames, dtype=torch.uint8, device="cuda")
    need = plan.workspace_size(frames)
    ws = torch.full((need + (1 << 20),), 255, dtype=torch.uint8, device="cuda")
    method = ck.MinSum(max_iterations=3)
    st = _lib.lib().ck_ldpc_decode(plan.handle, x.data_ptr(), out.data_ptr(), frames, n, *_rule_args(method), 3, 1,
                                   iters.data_ptr(), valid.data_ptr(), bits.data_ptr(), k, ws.data_ptr(), need,
                                   _device.stream_of(_device.wrap(x)))  # fmt: skip
    _lib.check(st, "decode")
    want = oracle.decode(llrs, (row_ptr, cols, N), k=k, scale=method.scale, offset=method.offset, max_iterations=3,
                         early_stop=True)  # fmt: skip
    got = [a.cpu().numpy() for a in (bits, out, valid, iters)]
    for g, w, what in zip(got, want, ("bits", "llrs", "valid", "iterations"), strict=True):
        np.testing.assert_array_equal(g, w, err_msg=what)
    assert bool((ws[need:] == 255).all()), "wrote past the workspace"
    return plan, need


# The 32-row groups' padded tables leave less than half of N, the row pointers alone the whole posterior; rows of
# 4, 3, 2 to 4, 12 and 24 edges.
CASES = [(32400, 16200, 3, 2), (30000, 15000, 2, 155), (20000, 16200, 5, 1), (32400, 16200, 10, 2), (32400, 16200, 22, 1)]


@pytest.mark.parametrize("N,m,weight,frames", CASES)
@pytest.mark.parametrize("placement", [0, 1, 2])
def test_posterior_in_shared_memory_without_row_groups(N, m, weight, frames, placement):
    check_serial(N, m, weight, frames, placement)


# Layers of one row whose 32-row groups would fit: 32 times the rows' state.
@pytest.mark.parametrize("N,m,weight,frames", [(16200, 9000, 3, 3), (2000, 1000, 3, 40), (600, 66, 2, 300)])
@pytest.mark.parametrize("placement", [0, 2])
def test_state_is_that_of_the_rows(N, m, weight, frames, placement):
    _, need = check_serial(N, m, weight, frames, placement)
    assert need <= 512 + frames * 2 * 12 * (m + 32)


@pytest.mark.parametrize("N,m,weight,threads", [(130, 66, 2, 1024), (4999, 2500, 3, 1024), (5000, 2500, 3, 768), (1000, 250, 3, 512)])
def test_short_codes_take_the_csr_rows(N, m, weight, threads):
    """Rows of up to 8 edges below N = 5000 run the CSR rows (up to 1024
    threads per frame; the 32-row groups cut a set shape to theirs)."""
    import commkit_gb300 as ck

    row_ptr, cols = staircase_rows(N, m, weight, seed=1)
    checks = np.repeat(np.arange(m, dtype=np.int32), np.diff(row_ptr))
    plan = ck.LDPCCode(checks, cols, m, N)._plan(0)
    assert plan.info["quasi_cyclic"] == 0
    plan.set_launch(1024, 0, 0)
    assert plan.resolved_launch()[0] == threads
