"""rl_radiosity_solve's row sums (quads read over the rows' ends) against
rl_radiosity_step's (entry by entry at the ends), bit for bit: rows that start
at every offset within a quad, empty rows, a matrix whose last quad is cut by
the end of its arrays, iterates that fit in shared memory and that do not,
and columns that are not 16-byte aligned."""
import ctypes as C

import numpy as np
import pytest

from relight_b200 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,shift", [(1, 0), (3, 0), (65, 0), (700, 0), (700, 1), (4800, 0), (19200, 0), (19200, 1)])
def test_solve_matches_row_steps(cuda, n, shift):
    import torch
    rng = np.random.default_rng(n)
    lens = rng.integers(0, 9, n)
    lens[rng.random(n) < 0.2] = 0
    big = rng.choice(n, min(n, 12), replace=False)
    lens[big] = rng.integers(100, 1100, len(big))
    lens[-1] = 5
    row = np.zeros(n + 1, np.int64)
    row[1:] = np.cumsum(lens)
    nnz = int(row[-1])
    cols = rng.integers(0, n, nnz).astype(np.int32)
    vals = (rng.random(nnz) / 1000).astype(np.float32)
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    dr = T(row)
    dc = T(np.concatenate([np.zeros(shift, np.int32), cols]))[shift:]
    dv = T(np.concatenate([np.zeros(shift, np.float32), vals]))[shift:]
    E, rho = T(rng.random((n, 3)).astype(np.float32)), T(rng.random((n, 3)).astype(np.float32))
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    L = _abi.lib()
    got = torch.empty_like(E)
    _abi.check(L.rl_radiosity_solve(n, P(dr), P(dc), P(dv), P(E), P(rho), 4, P(got), None))
    B, Bn = E.clone(), torch.empty_like(E)
    for _ in range(4):
        _abi.check(L.rl_radiosity_step(0, n, P(dr), P(dc), P(dv), P(E), P(rho), P(B), P(Bn), None))
        B, Bn = Bn, B
    assert torch.equal(got.view(torch.int32), B.view(torch.int32))


def test_solve_under_capture(cuda):
    """A captured solve replays what the direct call computes."""
    import torch
    n = 300
    rng = np.random.default_rng(1)
    row = torch.arange(0, 8 * (n + 1), 8, dtype=torch.int64, device="cuda")
    cols = torch.from_numpy(rng.integers(0, n, 8 * n).astype(np.int32)).cuda()
    vals = torch.from_numpy((rng.random(8 * n) / 10).astype(np.float32)).cuda()
    E, rho = torch.rand(n, 3, device="cuda"), torch.rand(n, 3, device="cuda")
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    L = _abi.lib()
    want, got = torch.empty_like(E), torch.zeros_like(E)
    _abi.check(L.rl_radiosity_solve_noalloc(n, P(row), P(cols), P(vals), P(E), P(rho), 7, P(want), None))
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _abi.check(L.rl_radiosity_solve_noalloc(n, P(row), P(cols), P(vals), P(E), P(rho), 7, P(got),
                                                torch.cuda.current_stream().cuda_stream))
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
