"""Sum-product decoding in the register form (two lanes per row, messages in
registers) against the table-driven kernel, bit for bit: liftings around its
16-row warps, rows of two, odd and many edges, one frame, a
block per frame and several waves."""

from __future__ import annotations

import numpy as np
import pytest

from commkit_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# mb, nb, Z, information column weights, frames.
CASES = [
    (4, 8, 2, 2, 1),
    (3, 7, 15, 2, 5),
    (5, 11, 16, 3, 33),
    (6, 12, 17, 3, 153),
    (12, 24, 54, 4, 5200),
    (6, 24, 96, 3, 1300),
    (4, 30, 31, 4, 64),  # rows of 27 edges
    (16, 48, 8, 3, 300),  # about the most edge slots
    (4, 9, 256, 2, 40),  # the most threads
    (4, 9, 257, 2, 40),  # beyond them
]


def _run(base, z, frames):
    import torch

    import commkit_gb300 as ck
    from commkit_gb300 import _lib

    rng = np.random.default_rng(3)
    got = []
    for mode in (_lib.CK_LDPC_SPECIALISE_OFF, _lib.CK_LDPC_SPECIALISE_AUTO):
        code = ck.LDPCCode.quasi_cyclic(base, lifting=z)
        code._plan(0).set_specialise(mode)
        if not got:
            llrs = (2.0 + 2.2 * rng.standard_normal((frames, code.n))).astype(np.float32)
            llrs[0, :6] = [0.0, -0.0, np.inf, -np.inf, 1e30, np.nan]
            x = torch.from_numpy(llrs).cuda()
        out = []
        for method in (ck.SumProduct(max_iterations=7), ck.SumProduct(max_iterations=3, early_stop=False)):
            ws = torch.full((code._plan(0).workspace_size(frames, _lib.CK_LDPC_SUM_PRODUCT),), 255, dtype=torch.uint8,
                            device="cuda")  # fmt: skip
            for r in (ck.decode(x, code=code, method=method), ck.decode(x, code=code, method=method, workspace=ws)):
                out += [r.bits, r.llrs, r.valid, r.iterations]
        got.append([o.cpu().numpy() for o in out])
    for want, have in zip(*got, strict=True):
        if want.dtype == np.float32:
            want, have = want.view(np.uint32), have.view(np.uint32)
        np.testing.assert_array_equal(have, want)


@pytest.mark.parametrize("mb,nb,z,weight,frames", CASES)
def test_equals_table_kernel(mb, nb, z, weight, frames):
    _run(W.dual_diagonal_base(mb, nb, z, (weight,) * (nb - mb), seed=z), z, frames)


def test_row_of_two_edges():
    base = W.dual_diagonal_base(6, 12, 17, (3,) * 6, seed=1)
    base[4, :6] = -1
    _run(base, 17, 40)


def test_no_workspace_for_messages_in_registers():
    """The register form keeps nothing in device memory, also for a code
    whose messages the table-driven kernel keeps there; a plan whose
    specialisation is turned off asks for that kernel's workspace anew."""
    import torch

    import commkit_gb300 as ck
    from commkit_gb300 import _lib

    rng = np.random.default_rng(8)
    base = np.full((8, 40), -1, np.int64)  # rows of 16: 64 edge slots per lane, 25,600 messages
    for i in range(8):
        base[i, (5 * i + np.arange(16)) % 40] = rng.integers(0, 200, 16)
    code = ck.LDPCCode.quasi_cyclic(base, lifting=200)
    plan = code._plan(0)
    assert plan.workspace_size(300, _lib.CK_LDPC_SUM_PRODUCT) <= 512
    x = torch.from_numpy((1.5 + 1.7 * rng.standard_normal((300, code.n))).astype(np.float32)).cuda()
    method = ck.SumProduct(max_iterations=4)
    ws = torch.full((512,), 255, dtype=torch.uint8, device="cuda")
    got = [ck.decode(x, code=code, method=method), ck.decode(x, code=code, method=method, workspace=ws)]
    plan.set_specialise(_lib.CK_LDPC_SPECIALISE_OFF)
    assert plan.workspace_size(300, _lib.CK_LDPC_SUM_PRODUCT) >= 152 * 4 * 25600
    want = ck.decode(x, code=code, method=method)
    for g in got:
        for name in ("bits", "llrs", "valid", "iterations"):
            np.testing.assert_array_equal(getattr(g, name).cpu().numpy(), getattr(want, name).cpu().numpy(), err_msg=name)


@pytest.mark.parametrize("rule", ["sum_product", "min_sum"])
def test_first_decode_inside_a_capture(rule):
    """The first decode of a plan, which compiles its kernel, recorded in a
    graph: the replay gives what a decode outside gives."""
    import torch

    import commkit_gb300 as ck

    base = W.dual_diagonal_base(5, 13, 24, (3,) * 8, seed=11)
    code = ck.LDPCCode.quasi_cyclic(base, lifting=24)
    code._plan(0)  # plans allocate their tables outside captures
    method = (ck.SumProduct if rule == "sum_product" else ck.MinSum)(max_iterations=8)
    x = torch.from_numpy((1.2 + 1.5 * np.random.default_rng(9).standard_normal((40, code.n))).astype(np.float32)).cuda()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        r = ck.decode(x, code=code, method=method)
    graph.replay()
    torch.cuda.synchronize()
    want = ck.decode(x, code=code, method=method)
    for name in ("bits", "llrs", "valid", "iterations"):
        np.testing.assert_array_equal(getattr(r, name).cpu().numpy(), getattr(want, name).cpu().numpy(), err_msg=name)


@pytest.mark.parametrize("rule", [0, 1])
def test_resolved_launch_can_be_set(rule):
    """The reported shape is one kernel's, which setting it selects."""
    import torch

    import commkit_gb300 as ck

    code = ck.LDPCCode.quasi_cyclic(W.dual_diagonal_base(5, 13, 72, (3,) * 8, seed=13), lifting=72)
    plan = code._plan(0)
    method = ck.MinSum(max_iterations=5) if rule == 0 else ck.SumProduct(max_iterations=5)
    x = torch.from_numpy((1.2 + 1.5 * np.random.default_rng(9).standard_normal((70, code.n))).astype(np.float32)).cuda()
    want = ck.decode(x, code=code, method=method)
    shape = plan.resolved_launch(rule)
    plan.set_launch(*shape)
    assert plan.resolved_launch(rule) == shape
    got = ck.decode(x, code=code, method=method)
    for name in ("bits", "llrs", "valid", "iterations"):
        np.testing.assert_array_equal(getattr(got, name).cpu().numpy(), getattr(want, name).cpu().numpy(), err_msg=name)
