"""Sum-product decoding of codes without circulants whose posterior is in
shared memory: a frame per SM takes more threads than two do, with the same
bits.  Batches around a frame per SM, layers shorter and longer than a block,
rows of any degree."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_ell import staircase_code

pytestmark = pytest.mark.gpu

# N, m, column weight, punctured (rows of 4 to 26 edges, the last of 32 and
# more; N = 40000 holds one frame per SM).
CASES = [(24, 12, 2, 0), (1999, 777, 3, 5), (16200, 9000, 3, 0), (9000, 1000, 3, 0), (40000, 20000, 3, 1),
         (6000, 500, 3, 0)]  # fmt: skip


@pytest.mark.parametrize("N,m,weight,punctured", CASES)
def test_batches_equal_a_set_shape(N, m, weight, punctured):
    import torch

    import commkit_gb300 as ck

    code = staircase_code(ck, N, m, weight, seed=N + m, punctured=punctured)
    plan = code._plan(0)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(7)
    llrs = (2.0 + 2.0 * rng.standard_normal((sms + 1, code.n))).astype(np.float32)
    llrs[0, :8] = [0.0, -0.0, np.inf, -np.inf, 1e30, -1e30, 1e-38, -1e-38]
    x = torch.from_numpy(llrs).cuda()
    method = ck.SumProduct(max_iterations=3)
    plan.set_launch(64)
    want = ck.decode(x, code=code, method=method)
    plan.set_launch()
    for frames in (1, sms, sms + 1):
        got = ck.decode(x[:frames], code=code, method=method)
        for what in ("bits", "llrs", "valid", "iterations"):
            g, w = (getattr(r, what)[:frames].cpu().numpy() for r in (got, want))
            np.testing.assert_array_equal(g.view(np.uint8), w.view(np.uint8), err_msg=f"{what}, {frames} frames")
