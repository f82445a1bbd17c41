"""The two streams of an objective: the fluence-gradient products run beside the
VOI ones.  What they share must not: a problem whose D is A itself gives what it
gives with a copy, bit for bit, and a problem without fluence-gradient rows what
it gives with empty ones."""
import numpy as np
import pytest

from fastdose_b200 import optimize

pytestmark = pytest.mark.gpu


def _csr(rng, rows, cols, per_row):
    counts = rng.integers(0, 2 * per_row, rows)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(cols, c, replace=False)) for c in counts]).astype(np.int64)
    return off, col, (rng.random(len(col)) * 0.05).astype(np.float32)


def _problem(ctx, A, AT, D, DT, rows, seed):
    rng = np.random.default_rng(seed)
    n_ptv = rows // 3
    return optimize.Problem(ctx, A, AT, D, DT, n_ptv, rows - n_ptv, np.full(rows, 1.05), rng.random(rows),
                            np.ones(n_ptv), np.ones(n_ptv), 0.1 * rng.random(rows - n_ptv), 1.0, 0.1)


def _results(P, cols, graph):
    import torch

    P.set_graph(graph)
    x = torch.rand(cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7))
    v, g = P.eval_grad(x)
    go = np.linspace(0, cols, 9).astype(np.int64)
    b = P.boo(go, np.full(8, 0.05, np.float32), x, 1e-3, 12, change_trigger=5)
    q = P.polish(x, 1e-3, 8)
    return [np.float64([v, P.eval_g(x)])] + [np.asarray(a.cpu() if hasattr(a, "cpu") else a)
                                             for a in (g, b["x"], b["v"], b["loss"], b["nrm"], q["x"], q["loss"])]


# x of 900 floats is gathered from shared memory; 60000 are scaled into the matrix's own buffer
@pytest.mark.parametrize("cols,vt", [(900, "f32"), (60000, "f16")])
@pytest.mark.parametrize("graph", [True, False])
def test_d_may_be_the_matrix_itself(ctx, graph, cols, vt):
    rows = 9000
    off, col, val = _csr(np.random.default_rng(3), rows, cols, 60)
    ms = [optimize.Matrix.from_csr(ctx, off, col, val, cols, value_type=vt, index_format="packed16") for _ in range(2)]
    ts = [m.transpose() for m in ms]
    apart = _results(_problem(ctx, ms[0], ts[0], ms[1], ts[1], rows, 1), cols, graph)
    for _ in range(5):
        same = _results(_problem(ctx, ms[0], ts[0], ms[0], ts[0], rows, 1), cols, graph)
        for a, b in zip(apart, same):
            np.testing.assert_array_equal(a, b)


def test_no_fluence_gradient_rows(ctx):
    rows, cols = 5000, 700
    off, col, val = _csr(np.random.default_rng(4), rows, cols, 40)
    A = optimize.Matrix.from_csr(ctx, off, col, val, cols)
    AT = A.transpose()
    out = []
    for m, graph in ((0, True), (0, False), (6, True)):
        D = optimize.Matrix.from_csr(ctx, np.zeros(m + 1, np.int64), np.zeros(0, np.int64), np.zeros(0, np.float32), cols)
        out.append(_results(_problem(ctx, A, AT, D, D.transpose(), rows, 2), cols, graph))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
