"""The one-launch CSR factorisation and triangular solves at their edges.

Rows are handed out in blocks (256 of them in the factorisation, 1024 in the
triangular solves) and solved in order of their dependencies, four terms of a
row at a time.  The matrices have one row fewer and one more than a block of
either kind, rows of no, four and five and many lower entries, an empty row,
and chains that cross every block.  The oracle's MIC(0)-PCG runs the
same recurrences; its dot products sum in another order, so the iterates differ
by rounding, and both stop at a residual of 1e-11 max|b|: they agree to that
times the inverse's norm, at most 10 for diagonals that exceed the row's other
entries by 0.1, here 1e-9 of the largest entry with a factor of ten to spare."""
import numpy as np
import pytest

from libwetcloth_b200 import _capi
from oracle import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _matrix(n, kind, seed=0):
    rng = np.random.default_rng(seed)
    pairs = set()
    if kind == "chain":  # every row waits for the one before
        pairs |= {(i, i - 1) for i in range(1, n)}
    elif kind == "wide":  # 0 to 8 lower entries a row
        for i in range(n):
            for j in rng.choice(i, min(i, i % 9), replace=False) if i else ():
                pairs.add((i, int(j)))
    else:  # "arrow": the last rows hold an entry of every fifth column
        pairs |= {(i, i - 1) for i in range(1, n) if i % 3}
        for i in range(max(1, n - 2), n):
            pairs |= {(i, j) for j in range(0, i, 5)}
    rows = [{} for _ in range(n)]
    empty = n // 2 if n > 2 else -1
    for i, j in pairs:
        if empty not in (i, j):
            rows[i][j] = rows[j][i] = -rng.uniform(0.2, 1.0)
    start, col, val = [0], [], []
    for i, r in enumerate(rows):
        if i != empty:
            r[i] = sum(abs(v) for v in r.values()) + rng.uniform(0.1, 1.0)
        for j in sorted(r):
            col.append(j)
            val.append(r[j])
        start.append(len(col))
    b = rng.standard_normal(n)
    if empty >= 0:
        b[empty] = 0.0
    return np.array(start, np.int64), np.array(col, np.int64), np.array(val), b


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 257, 513, 1023, 1024, 1025, 2049, 5000])
@pytest.mark.parametrize("kind", ["chain", "wide", "arrow"])
def test_dataflow_edges_match_oracle(n, kind, wcg):
    rs, col, val, b = _matrix(n, kind, n)
    xg, resg, itg, st = _capi.pcg_solve_csr(rs, col, val, b, TOL, 500)
    xo, ok, ito, _ = oracle.pcg_solve(rs, col, val, b, TOL, 500)
    assert ok and st == _capi.WCG_OK and abs(itg - ito) <= 1
    assert resg <= TOL * np.abs(b).max()
    assert np.abs(xg - xo).max() <= 1e-9 * np.abs(xo).max()
    # the same bits again, on fresh buffers
    assert np.array_equal(xg, _capi.pcg_solve_csr(rs, col, val, b, TOL, 500)[0])


def _band(n, w):
    """Symmetric, diagonally dominant, every row coupled to its w neighbours on
    either side."""
    rng = np.random.default_rng(n + w)
    off = np.zeros((n, 2 * w + 1))
    on = np.zeros(off.shape, bool)
    for d in range(1, w + 1):
        u = -rng.uniform(0.2, 1.0, n - d)
        off[d:, w - d], off[:n - d, w + d] = u, u
        on[d:, w - d] = on[:n - d, w + d] = True
    off[:, w] = np.abs(off).sum(1) + rng.uniform(0.1, 1.0, n)
    on[:, w] = True
    col = (np.arange(n)[:, None] + np.arange(-w, w + 1))[on]
    return np.concatenate([[0], np.cumsum(on.sum(1))]), col, off[on], rng.standard_normal(n)


def test_long_chain_of_wide_rows(wcg):
    """A band of 24 over 60 000 rows: every column waits for the one before, and
    the last ones, resident from the start, wait for seconds.  The band has no
    dropped entries, so the factor is the Cholesky factor: one iteration, as
    the oracle takes."""
    rs, col, val, b = _band(60000, 24)
    xg, resg, itg, st = _capi.pcg_solve_csr(rs, col, val, b, TOL, 20)
    xo, ok, ito, _ = oracle.pcg_solve(rs, col, val, b, TOL, 20)
    assert ok and st == _capi.WCG_OK and itg == ito
    assert resg <= TOL * np.abs(b).max()
    assert np.abs(xg - xo).max() <= 1e-9 * np.abs(xo).max()


def test_device_memory_of_a_solve(wcg):
    """The factor and its transpose take the entries right of the diagonal, not
    all: per entry of the matrix 12 bytes, per entry of the factor 20, per row
    80 and a little (a pollster sees the least free memory while the solve
    runs; 10 % for granularity)."""
    torch = pytest.importorskip("torch")
    import threading
    import time
    blocks, w = 6000, 80  # dense blocks: chains of 80 rows
    n = blocks * w
    rng = np.random.default_rng(0)
    B = -rng.uniform(0.2, 1.0, (w, w))
    B = B + B.T
    np.fill_diagonal(B, np.abs(B).sum(1) + 1.0)
    val = np.tile(B.reshape(-1), blocks)
    col = (np.arange(blocks, dtype=np.int32)[:, None, None] * w +
           np.arange(w, dtype=np.int32)[None, None] + np.zeros((1, w, 1), np.int32)).reshape(-1)
    rs = np.arange(n + 1, dtype=np.int32) * w
    b = rng.standard_normal(n)
    _capi.pcg_solve_csr(rs[:w + 1], col[:w * w], val[:w * w], b[:w], TOL, 20)  # the context
    free, _ = torch.cuda.mem_get_info()
    least, done = [free], threading.Event()

    def watch():
        while not done.is_set():
            least[0] = min(least[0], torch.cuda.mem_get_info()[0])
            time.sleep(5e-4)

    t = threading.Thread(target=watch)
    t.start()
    try:
        x, res, it, st = _capi.pcg_solve_csr(rs, col, val, b, TOL, 20)
    finally:
        done.set()
        t.join()
    assert st == _capi.WCG_OK and res <= TOL * np.abs(b).max()
    nnz, nu = n * w, blocks * w * (w - 1) // 2
    used = free - least[0]
    assert 0.9 * (12 * nnz + 20 * nu) <= used <= 1.1 * (12 * nnz + 20 * nu + 84 * n)
