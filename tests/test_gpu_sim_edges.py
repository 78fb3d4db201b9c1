"""The simulation's random bits and error counts at the edges of their wide
paths: lengths around a word and a Philox block, outputs at every alignment,
rows whose lengths or addresses rule the wide loads out."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_sim import bits_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 31, 32, 33, 127, 128, 129, 4095, 100_003])
@pytest.mark.parametrize("offset", [0, 1, 4, 16])
def test_random_bits(count, offset):
    import torch

    from commkit_gb300 import _device, _lib

    buf = torch.full((count + offset + 40,), 7, dtype=torch.int8, device="cuda")
    st = _device.stream_of(_device.wrap(buf))
    _lib.check(_lib.lib().ck_random_bits(buf.data_ptr() + offset, count, 11, 5, st), "random bits")
    got = buf.cpu().numpy()
    np.testing.assert_array_equal(got[offset : offset + count], bits_np(count, 11, 5))
    assert (got[:offset] == 7).all() and (got[offset + count :] == 7).all()


@pytest.mark.parametrize("k,n", [(1, 1), (4, 8), (648, 1296), (1023, 2048), (1024, 2047), (2000, 5000)])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("frames", [1, 203, 1300])
def test_error_counts(k, n, offset, frames):
    import torch

    from commkit_gb300 import _device, _lib

    rng = np.random.default_rng(k + frames)
    info = rng.integers(0, 2, (frames, k)).astype(np.int8)
    decoded = info ^ (rng.random((frames, k)) < 0.01).astype(np.int8)
    decoded[::3] = info[::3]
    sent = rng.integers(0, 2, (frames, n)).astype(np.int8)
    llr = (rng.standard_normal((frames, n)) * 3).astype(np.float32)
    llr.reshape(-1)[: 4 if n * frames > 4 else 1] = [np.nan, -0.0, -np.inf, np.inf][: 4 if n * frames > 4 else 1]
    valid = rng.integers(0, 2, frames).astype(np.uint8)
    iters = rng.integers(-1, 50, frames).astype(np.int32)

    def dev(a):  # the array `offset` elements into a buffer
        buf = torch.zeros(a.size + 8, dtype=torch.from_numpy(a).dtype, device="cuda")
        view = buf[offset : offset + a.size]
        view.copy_(torch.from_numpy(a.reshape(-1)))
        return view

    arrays = [dev(a) for a in (info, decoded, llr, sent)]
    v, it = torch.from_numpy(valid).cuda(), torch.from_numpy(iters).cuda()
    counts = torch.full((7,), 5, dtype=torch.int64, device="cuda")
    st = _device.stream_of(_device.wrap(counts))
    _lib.check(_lib.lib().ck_count_errors(*(a.data_ptr() for a in arrays), frames, k, n, v.data_ptr(), it.data_ptr(),
                                          counts.data_ptr(), st), "error counts")  # fmt: skip
    errors = (info != decoded).sum(1)
    want = [frames, errors.sum(), (errors > 0).sum(), ((llr < 0) != (sent != 0)).sum(), (valid == 0).sum(),
            ((errors > 0) & (valid != 0)).sum(), np.maximum(iters, 0).sum()]  # fmt: skip
    np.testing.assert_array_equal(counts.cpu().numpy(), np.array(want) + 5)
