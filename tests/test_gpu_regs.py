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



# The kernels that launches run, by the profiler's names.  In a process of its
# own that keeps its codes: the profiler names kernels by handles, which a
# destroyed plan's library leaves to the next.
PROFILED = """
import sys
import numpy as np, torch
from torch.profiler import ProfilerActivity, profile
import commkit_gb300 as ck
from commkit_gb300 import _device, _lib, workloads as W

def kernels(f):
    f()
    for _ in range(2):  # a process's first profile may come back empty
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            f()
            torch.cuda.synchronize()
    names = {e.name for e in p.events()}
    if not any("kernel" in n or n.startswith("ck_ldpc") for n in names):
        print("no profiler")
        sys.exit(0)
    return names
"""


def _profiled(body: str) -> None:
    import subprocess
    import sys
    from pathlib import Path

    r = subprocess.run([sys.executable, "-c", PROFILED + body], capture_output=True, text=True, timeout=600,
                       cwd=Path(__file__).resolve().parents[1])  # fmt: skip
    assert r.returncode == 0, r.stdout + r.stderr
    if "no profiler" in r.stdout:
        pytest.skip("no profiler")


def test_form_by_waves():
    """The register form up to the waves that its width and row length bear,
    the shared form beyond (both bit-identical): 18 or 12 information columns
    of weight 4 or 3, so rows of 13.8 and 4.9."""
    _profiled("""
codes = []
sms = torch.cuda.get_device_properties(0).multi_processor_count
for mb, z, weight, waves in ((12, 160, 3, 1), (12, 256, 3, 1), (6, 160, 4, 2), (12, 54, 3, 4), (6, 64, 4, 8), (12, 16, 3, 8)):
    base = W.dual_diagonal_base(mb, 24, z, (weight,) * (24 - mb), seed=z)
    code = ck.LDPCCode.quasi_cyclic(base, lifting=z)
    codes.append(code)
    slots = sum((int(d) + 1) // 2 for d in (base >= 0).sum(1))
    per_sm = min(max(65536 // ((2 * slots + 40 + 7) // 8 * 8 * ((z + 15) // 16 * 32)), 1), 16)
    for w, registers in ((waves, True), (waves + 0.3, False)):
        x = torch.full((int(w * sms * per_sm), code.n), 4.0, device="cuda")
        names = kernels(lambda: ck.decode(x, code=code, method=ck.MinSum(max_iterations=2)))
        assert ("ck_ldpc_code_r3" in names) == registers, (mb, z, w, names)
""")


def test_a_decode_compiles_only_the_placements_it_runs():
    """With specialisation required, the fixed-scratch entry runs the kernel a
    decode compiled, and the table-driven one (the same bits) after a launch
    of another placement that none has run."""
    _profiled("""
code = ck.LDPCCode.quasi_cyclic(W.dual_diagonal_base(5, 13, 40, (3,) * 8, seed=12), lifting=40)
plan = code._plan(0)
plan.set_specialise(_lib.CK_LDPC_SPECIALISE_ON)
x = torch.from_numpy((1.2 + 1.5 * np.random.default_rng(9).standard_normal((30, code.n))).astype(np.float32)).cuda()
want = ck.decode(x, code=code, method=ck.MinSum(max_iterations=6))
assert plan.specialisation()[1] == 1
out, bits = torch.empty_like(x), torch.empty((30, code.k), dtype=torch.int8, device="cuda")
it, ok = torch.empty(30, dtype=torch.int32, device="cuda"), torch.empty(30, dtype=torch.uint8, device="cuda")

def static():
    out.zero_()
    names = kernels(lambda: _lib.check(_lib.lib().ck_ldpc_decode_static(
        plan.handle, x.data_ptr(), out.data_ptr(), 30, code.n, 0, 0.875, 0.0, 6, 1, it.data_ptr(), ok.data_ptr(),
        bits.data_ptr(), code.k, _device.stream_of(_device.wrap(x))), "static"))
    np.testing.assert_array_equal(out.cpu().numpy(), want.llrs.cpu().numpy())
    np.testing.assert_array_equal(it.cpu().numpy(), want.iterations.cpu().numpy().reshape(-1))
    return {k for k in names if k.startswith("ck_ldpc_code")}

assert static() == {"ck_ldpc_code_r3"}
plan.set_launch(64, 2, _lib.CK_LDPC_PLACE_GLOBAL)
assert static() == set()
ck.decode(x, code=code, method=ck.MinSum(max_iterations=6))
assert static() == {"ck_ldpc_code_r0"}
""")
