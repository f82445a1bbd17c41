"""Products over rows of a constant length around the lane (8), slice (32) and
chunk (256 nonzeros) sizes of the stream kernel, with runs of empty rows, in the
forms a matrix is stored in: x in shared memory, and x in global memory with
short rows (a lane's elements consecutive) or long ones (interleaved).  A large x in
shared memory (scaled by a launch of its own, and interleaved with 16-bit values and
long rows) has a test of its own: it takes a matrix of more bytes than its copies.

Tolerance: a row of n nonzeros is a sum in FP32 of n products in some order, so
it is within (n + 2) 2^-24 of its |A||x| sum."""
import numpy as np
import pytest

from fastdose_b200 import optimize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [900, 60000])
@pytest.mark.parametrize("length", [1, 2, 7, 8, 9, 31, 33, 63, 64, 65, 255, 256, 257, 700])
def test_rows_of_one_length(ctx, cols, length):
    import torch

    rng = np.random.default_rng(length)
    rows = max(40, 40000 // length) + 3
    counts = np.full(rows, length, np.int64)
    counts[rng.random(rows) < 0.2] = 0
    counts[:2] = 0
    counts[-1] = 0
    counts[rows // 2] = min(cols, 5 * length + 3)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    # ascending columns: a random start and random gaps that stay inside
    col = np.concatenate([np.sort(rng.choice(cols, c, replace=False)) for c in counts]).astype(np.int64)
    val = (rng.random(len(col)) - 0.3).astype(np.float32)
    x = rng.standard_normal(cols).astype(np.float32)
    row = np.repeat(np.arange(rows), counts)
    for vt, fmt in (("f32", "i32"), ("f32", "packed16"), ("f16", "packed16"), ("bf16", "i32")):
        M = optimize.Matrix.from_csr(ctx, off, col, val, cols, value_type=vt, index_format=fmt)
        o, c, v = M.to_host()
        np.testing.assert_array_equal(o, off)
        np.testing.assert_array_equal(c, col)
        y = M.spmv(torch.from_numpy(x).cuda()).cpu().numpy()
        p = v.astype(np.float64) * x[col]
        ref = np.bincount(row, p, rows)
        bound = np.bincount(row, np.abs(p), rows)
        # 16-bit values: x is scaled by the column's scale, one more rounding each
        assert np.all(np.abs(y - ref) <= (counts + 4) * 2.0 ** -24 * bound)
        assert np.all(y[counts == 0] == 0)
        T = M.transpose()
        z = rng.standard_normal(rows).astype(np.float32)
        yt = T.spmv(torch.from_numpy(z).cuda()).cpu().numpy()
        q = v.astype(np.float64) * z[row]
        n_col = np.bincount(col, minlength=cols)
        # 16-bit values: the row's scale times a sum of the values without it, two more roundings
        assert np.all(np.abs(yt - np.bincount(col, q, cols)) <= (n_col + 5) * 2.0 ** -24 * np.bincount(col, np.abs(q), cols))
        for a, b in zip(T.transpose().to_host(), (o, c, v)):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("per", [20, 95, 120, 255, 260, 900])
@pytest.mark.parametrize("vt,fmt", [("f16", "packed16"), ("bf16", "i32"), ("f32", "packed16")])
def test_large_x_in_shared_memory(ctx, vt, fmt, per):
    import torch

    rng = np.random.default_rng(per)
    cols, rows = 20000, 3_200_000 // per
    counts = np.minimum(rng.poisson(per, rows), cols)
    counts[rng.random(rows) < 0.05] = 0
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    row = np.repeat(np.arange(rows), counts)
    gap = (cols // (counts + 1))[row]  # one column in each of the row's gaps
    col = (np.arange(off[-1]) - off[row]) * gap + rng.integers(0, 1 << 30, off[-1]) % gap
    val = (rng.random(off[-1]) - 0.3).astype(np.float32)
    M = optimize.Matrix.from_csr(ctx, off, col, val, cols, value_type=vt, index_format=fmt)
    assert M.info()["x_in_shared"]
    x = rng.standard_normal(cols).astype(np.float32)
    _, c, v = M.to_host()
    np.testing.assert_array_equal(c, col)
    y = M.spmv(torch.from_numpy(x).cuda()).cpu().numpy()
    p = v.astype(np.float64) * x[col]
    assert np.all(np.abs(y - np.bincount(row, p, rows)) <= (counts + 4) * 2.0 ** -24 * np.bincount(row, np.abs(p), rows))
    np.testing.assert_array_equal(M.spmv(torch.from_numpy(x).cuda()).cpu().numpy(), y)


def test_device_bytes_count_the_rows_a_product_clears(ctx):
    """Empty rows are in the list each product reads: 4 bytes a row."""
    rng = np.random.default_rng(2)
    col = np.sort(rng.choice(900, 300, replace=False)).astype(np.int64)
    val = np.ones(300, np.float32)
    size = []
    for empty in (0, 1000):
        off = np.concatenate([[0, 300], np.full(empty, 300)]).astype(np.int64)
        size.append(optimize.Matrix.from_csr(ctx, off, col, val, 900).info()["device_bytes"])
    assert size[1] - size[0] == 4 * 1000


def test_matrix_memory_waits_for_products_and_outlives_the_context():
    """A matrix is destroyed while its product runs on another stream, and after
    its context; its memory is not handed to the next matrix before that."""
    import torch

    from fastdose_b200 import api

    ctx = api.Context(0)
    A, AT = optimize.Matrix.synthetic(ctx, 200_000, 4000, 8000, 0.5, seed=5)
    x = torch.rand(4000, device="cuda")
    ref = A.spmv(x).clone()
    torch.cuda.synchronize()
    y = torch.empty_like(ref)
    s = torch.cuda.Stream()
    for _ in range(20):
        A.spmv(x, y, stream=s)
    A.close()
    B, BT = optimize.Matrix.synthetic(ctx, 200_000, 4000, 8000, 0.5, seed=6)
    s.synchronize()
    assert torch.equal(y, ref)
    ctx.close()
    for m in (AT, B, BT):
        m.close()
