"""The encode kernel that holds its rows in registers (padded dims 256, 512 and
1024, more than 8 rows a multiprocessor) against the one-row-per-warp kernel of
small inputs, which the oracle tests cover: the same bytes, at every bit width,
at ragged dims and row counts, for rows of every magnitude, zero, infinite and
NaN rows, and inputs and outputs that are not 16-byte aligned."""
import numpy as np
import pytest

import oracle as O
import turboquant as tq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [129, 131, 255, 256, 257, 384, 509, 512, 516, 770, 1001, 1020, 1024])
@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8, 9])
@pytest.mark.parametrize("extra", [1, 4])
def test_register_rows_equal_single_rows(cuda_ok, dim, bits, extra):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 40 * sms + extra
    rng = np.random.default_rng(dim * 10 + bits)
    X = (rng.standard_normal((n, dim)) * rng.uniform(1e-3, 1e3, (n, 1))).astype(np.float32)
    X[1], X[2, 1:], X[3], X[-1, :-1] = 0.0, 0.0, 1.0, 0.0
    X[5] *= 1e-30
    X[6] *= 1e18
    X[7, dim // 2] = np.inf
    X[8, dim - 1] = np.nan
    s = tq.TurboQuantSpace(dim, bits)
    x = torch.from_numpy(X).cuda()
    piece = 8 * sms
    want = torch.cat([s.encode_batch(x[i:i + piece]) for i in range(0, n, piece)])
    assert torch.equal(s.encode_batch(x), want)
    assert torch.equal(s.encode_batch(x[1:]), want[1:])  # odd dims: rows off 16 bytes
    rows = [0, 2, 3, n // 2, n - 2]
    np.testing.assert_array_equal(want[rows].cpu().numpy(), O.OracleSpace(dim, bits).encode_batch(X[rows]))
