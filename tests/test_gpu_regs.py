"""Min-sum batches of the register form (two lanes per row, messages and
columns in registers) against the CPU oracle, bit for bit: liftings around
its 16-row warps, rows of odd and even degree, codes at and above its edge
slots, batches of one frame, of a block per frame and of several waves."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from commkit_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# mb, nb, Z, information column weights, punctured, frames.
CASES = [
    (4, 8, 2, 2, 0, 1),
    (3, 7, 15, 2, 0, 5),
    (5, 11, 16, 3, 3, 33),
    (6, 12, 17, 3, 0, 153),
    (12, 24, 54, 4, 0, 700),
    (12, 24, 54, 4, 1, 5200),
    (6, 24, 96, 3, 0, 1300),
    (4, 30, 31, 4, 0, 64),  # rows of 27 edges
    (16, 48, 8, 3, 0, 300),  # 72 slots: about the limit
    (20, 60, 8, 3, 0, 300),  # beyond it
    (4, 9, 256, 2, 0, 40),
    (4, 9, 257, 2, 0, 40),  # beyond its threads
]


@pytest.mark.parametrize("mb,nb,z,weight,punctured,frames", CASES)
def test_circulant_codes_equal_oracle(mb, nb, z, weight, punctured, frames):
    import torch

    import commkit_gb300 as ck
    from commkit_gb300 import _device, _lib

    base = W.dual_diagonal_base(mb, nb, z, (weight,) * (nb - mb), seed=z)
    code = ck.LDPCCode.quasi_cyclic(base, lifting=z, punctured=punctured)
    rng = np.random.default_rng(3)
    llrs = (2.0 + 2.2 * rng.standard_normal((frames, code.n))).astype(np.float32)
    llrs[0, :6] = [0.0, -0.0, np.inf, -np.inf, 1e30, np.nan]
    x = torch.from_numpy(llrs).cuda()
    row_ptr, cols, _ = code._schedule
    for method in (ck.MinSum(max_iterations=9), ck.MinSum(scale=0.75, offset=0.05, max_iterations=3, early_stop=False)):
        want = oracle.decode(llrs, (row_ptr, cols, code.num_variables), k=code.k, scale=method.scale,
                             offset=method.offset, max_iterations=method.max_iterations,
                             early_stop=method.early_stop)  # fmt: skip
        # The caller's workspace as it comes: its header is not zeroed.
        ws = torch.full((code._plan(0).workspace_size(frames),), 255, dtype=torch.uint8, device="cuda")
        for r in (ck.decode(x, code=code, method=method), ck.decode(x, code=code, method=method, workspace=ws)):
            got = (r.bits, r.llrs, r.valid, r.iterations)
            for g, w, what in zip(got, want, ("bits", "llrs", "valid", "iterations"), strict=True):
                np.testing.assert_array_equal(g.cpu().numpy().reshape(w.shape), w, err_msg=what)
        wd = _device.wrap(ws)
        assert _lib.lib().ck_ldpc_workspace_status(wd.ptr, _device.stream_of(wd)) == _lib.CK_OK


def _kernels(f):
    """Names of the kernels that ``f`` launches, as the profiler sees them."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    f()
    for _ in range(2):  # a process's first profile may come back empty
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            f()
            torch.cuda.synchronize()
    return {e.name for e in p.events()}


# Information column weights 3 of 12 of 24 base columns (rows of 4.9) and 4 of 18 (13.8): short and long rows.
@pytest.mark.parametrize("mb,z,weight,waves,beyond", [
    (12, 160, 3, 1.0, 1.3),
    (12, 256, 3, 1.0, 1.3),
    (6, 160, 4, 2.0, 2.3),
    (12, 54, 3, 4.0, 4.3),
    (6, 64, 4, 8.0, 8.3),
    (12, 16, 3, 8.0, 8.3),
])  # fmt: skip
def test_form_by_waves(mb, z, weight, waves, beyond):
    """The register form up to the waves that its width and row length bear,
    the shared form beyond (both bit-identical)."""
    import torch

    import commkit_gb300 as ck

    base = W.dual_diagonal_base(mb, 24, z, (weight,) * (24 - mb), seed=z)
    code = ck.LDPCCode.quasi_cyclic(base, lifting=z)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    slots = sum((int(d) + 1) // 2 for d in (base >= 0).sum(1))
    threads = (z + 15) // 16 * 32
    per_sm = min(max(65536 // ((2 * slots + 40 + 7) // 8 * 8 * threads), 1), 16)
    names = {}
    for w in (waves, beyond):
        x = torch.full((int(w * sms * per_sm), code.n), 4.0, device="cuda")
        names[w] = _kernels(lambda: ck.decode(x, code=code, method=ck.MinSum(max_iterations=2)))
    if not any(k.startswith("ck_ldpc") for n in names.values() for k in n):
        pytest.skip("no profiler")
    assert "ck_ldpc_code_r3" in names[waves] and "ck_ldpc_code_r3" not in names[beyond]
