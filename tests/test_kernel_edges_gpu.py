"""Kernels at the sizes where their tiles, remainders and dispatch rules end,
against the oracle (bit for bit unless a test says otherwise)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 257, 1000])
@pytest.mark.parametrize("dim,pd,offset", [(1, 16, 0), (3, 16, 0), (4, 16, 0), (32, 32, 0), (33, 48, 0), (100, 112, 0),
                                           (64, 96, 0), (64, 64, 1)])
def test_encode_fp16_row_and_column_remainders(cuda, oracle_mod, n, dim, pd, offset):
    """32-row warps and 32-column chunks, padding wider than the rows' last
    chunk, and rows that do not start on a 16-byte boundary (offset floats)."""
    from fvgb300 import scan

    torch = cuda
    rng = np.random.default_rng(n * 131 + dim)
    x = (rng.standard_normal((n, dim)) * np.exp(rng.uniform(-8, 8, (n, 1)))).astype(np.float32)
    buf = torch.empty(n * dim + offset, device="cuda")
    xd = buf[offset:].view(n, dim)
    xd.copy_(torch.from_numpy(x))
    codes, norms = scan.encode_fp16(xd, pd)
    ref_codes, ref_norms = oracle_mod.encode_fp16_padded(x)
    got = codes.cpu().numpy().view(np.uint16)
    assert np.array_equal(got[:, :dim], ref_codes[:, :dim])
    assert not got[:, dim:].any()
    assert np.array_equal(norms.cpu().numpy().view(np.uint32), ref_norms.view(np.uint32))
