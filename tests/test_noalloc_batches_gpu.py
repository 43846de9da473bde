"""mvdr_bsr6_spmv_dot_noalloc at the edges of its batches of blocks, of its blocks of
rows and of the chunks of partial sums: y equal to the row's sum in order (products
of floats are exact in double), x.y within the rounding of its double sum."""
import ctypes as C

import numpy as np
import pytest
import torch

from multiviewdynrecon_b200 import abi, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 31, 33, 768 * 32, 768 * 32 + 1])
def test_rows_of_every_length(rows):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(rows)
    count = np.arange(rows) % 20  # 0 .. 19 blocks
    rowptr = np.concatenate([[0], np.cumsum(count)]).astype(np.int32)
    nnz = int(rowptr[-1])
    col = rng.integers(0, rows, nnz).astype(np.int32)
    blocks = rng.normal(size=(nnz, 6, 6)).astype(np.float32)
    x = rng.normal(size=(rows, 6)).astype(np.float32)
    y64 = np.zeros((rows, 6))
    for q in range(20):
        has = np.nonzero(count > q)[0]
        s = rowptr[has] + q
        for k in range(6):
            y64[has] += blocks[s, :, k].astype(np.float64) * x[col[s], k].astype(np.float64)[:, None]
    want = y64.astype(np.float32)
    # (from an odd float: no alignment beyond that of a float is needed)
    gb = torch.zeros(36 * nnz + 1, device="cuda")
    gb[1:] = torch.from_numpy(blocks.reshape(-1)).cuda()
    rp, ci, gx = (torch.from_numpy(a).cuda() for a in (rowptr, col, x.reshape(-1)))
    y, dot = torch.empty_like(gx), torch.empty(1, dtype=torch.float64, device="cuda")
    ptr = [C.c_void_p(t.data_ptr()) for t in (rp, ci, gb[1:], gx, y, dot)]
    st = lib().mvdr_bsr6_spmv_dot_noalloc(rows, nnz, *ptr, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == abi.MVDR_OK, lib().mvdr_last_error_string()
    assert np.array_equal(y.cpu().numpy().reshape(rows, 6), want)
    terms = x.astype(np.float64) * want.astype(np.float64)
    assert abs(dot.item() - terms.sum()) <= 2.0 ** -53 * terms.size * np.abs(terms).sum() * 2
