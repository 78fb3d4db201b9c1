"""The one-kernel accumulator encoder against a host encoder, at the edges of
its frame groups, residue tiles, chunks and vector widths."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def accumulator_code(ck, k: int, m: int, g: int, punctured: int, seed: int):
    """k information columns of three ones, parity column c with ones in rows
    c and c + g."""
    rng = np.random.default_rng(seed)
    rows = np.concatenate([rng.integers(0, m, 3 * k), np.arange(m)])  # and every row at least one
    cols = np.concatenate([np.repeat(np.arange(k), 3), rng.integers(0, k, m)])
    key = np.unique(rows.astype(np.int64) * k + cols)
    c = np.arange(m)
    checks = np.concatenate([key // k, c, c[c + g < m] + g])
    variables = np.concatenate([key % k, k + c, k + c[c + g < m]])
    return ck.LDPCCode(checks, variables, m, k + m, punctured)


def host_encode(code, g: int, info: np.ndarray) -> np.ndarray:
    k, m = code.k, code.num_checks
    s = np.zeros((info.shape[0], m), np.int64)
    e = code.variables < k
    np.add.at(s.T, code.checks[e], info[:, code.variables[e]].T)
    for j in range(g, m):
        s[:, j] += s[:, j - g]
    return np.concatenate([info, (s % 2).astype(np.int8)], 1)[:, : code.n]


# k, m, g, punctured, frames: one frame; groups of 32 and a remainder; chains
# of one step, of one residue, of residues below and above a tile, a block's
# threads and a warp; a last chain step that is partial; odd k, m and n.
CASES = [
    (16, 8, 1, 0, 1),
    (17, 9, 1, 1, 33),
    (64, 96, 96, 0, 70),
    (100, 61, 2, 0, 5),
    (513, 300, 31, 7, 31),
    (640, 333, 32, 0, 64),
    (648, 648, 54, 0, 203),
    (1001, 700, 33, 0, 3),
    (2048, 2400, 600, 3, 35),
    (8448, 17664, 384, 0, 37),
    (4000, 3001, 1, 0, 150),
    (32400, 32400, 1, 0, 2),
    (56000, 512, 1, 0, 3),
    (60000, 512, 64, 0, 3),
]


@pytest.mark.parametrize("k,m,g,punctured,frames", CASES)
def test_accumulator_codes_equal_host(k, m, g, punctured, frames):
    import torch

    import commkit_gb300 as ck
    from commkit_gb300.coding import encode_blocks

    code = accumulator_code(ck, k, m, g, punctured, seed=k + g)
    assert code._encoder.inverse is None and code._encoder.stride == min(g, m)
    info = np.random.default_rng(5).integers(0, 2, (frames, k), dtype=np.int8)
    want = host_encode(code, min(g, m), info)
    x = torch.from_numpy(info).cuda()
    np.testing.assert_array_equal(ck.encode(x, code=code).cpu().numpy(), want)
    np.testing.assert_array_equal(ck.encode(x.view(torch.uint8).reshape(-1), code=code).cpu().numpy(), want.reshape(-1))
    np.testing.assert_array_equal(ck.encode(x.long(), code=code).cpu().numpy(), want)
    # Unaligned rows: inputs and outputs one byte into a buffer.
    buf = torch.zeros(frames * k + 1, dtype=torch.int8, device="cuda")
    out = torch.full((frames * code.n + 1,), 9, dtype=torch.int8, device="cuda")
    buf[1:] = x.reshape(-1)
    encode_blocks(code, buf[1:].view(frames, k), out[1:].view(frames, code.n))
    np.testing.assert_array_equal(out[1:].cpu().numpy(), want.reshape(-1))
    assert int(out[0]) == 9
    for bad in (2, -1):
        y = x.clone()
        y[frames - 1, k - 1] = bad
        with pytest.raises(ValueError, match="0 or 1"):
            ck.encode(y, code=code)


# k, m, frames on both sides of the line between the byte-wise kernels and the one-kernel encoder.
@pytest.mark.parametrize("k,m,frames,few", [
    (9000, 5000, 1, True),
    (9000, 5000, 64, True),
    (9000, 5000, 65, False),
    (7200, 9000, 32, True),
    (7200, 9000, 33, False),
    (9000, 4999, 1, False),
    (6200, 7800, 1, False),
])  # fmt: skip
def test_few_frames_of_a_long_chain(k, m, frames, few):
    import torch
    from torch.profiler import ProfilerActivity, profile

    import commkit_gb300 as ck
    from commkit_gb300.coding import encode_blocks

    code = accumulator_code(ck, k, m, 1, 0, seed=k + m)
    info = np.random.default_rng(5).integers(0, 2, (frames, k), dtype=np.int8)
    x = torch.from_numpy(info).cuda()
    np.testing.assert_array_equal(encode_blocks(code, x).cpu().numpy(), host_encode(code, 1, info))
    for _ in range(2):  # a process's first profile may come back empty
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            encode_blocks(code, x)
            torch.cuda.synchronize()
    names = " ".join(e.name for e in p.events())
    if "_kernel" not in names:
        pytest.skip("no profiler")
    assert ("syndrome_kernel" in names) == few and ("encode_kernel" in names) != few


def test_more_bits_than_a_block_holds_go_straight_to_the_general_path(monkeypatch):
    """encode() allocates and calls nothing for the checking kernel where it
    cannot serve; just below, it serves."""
    import torch

    import commkit_gb300 as ck
    from commkit_gb300 import _lib

    lib = _lib.lib()
    calls = []
    checked = lib.ck_ldpc_encode_checked
    monkeypatch.setattr(lib, "ck_ldpc_encode_checked", lambda *a: (calls.append(a[2]), checked(*a))[1])
    for k, served in ((49376, True), (49377, False)):
        code = accumulator_code(ck, k, 600, 1, 0, seed=k)
        info = np.random.default_rng(6).integers(0, 2, (2, k), dtype=np.int8)
        calls.clear()
        got = ck.encode(torch.from_numpy(info).cuda(), code=code)
        np.testing.assert_array_equal(got.cpu().numpy(), host_encode(code, 1, info))
        assert (len(calls) == 1) == served
