"""Where device memory ends: the tables a solve can do without (K times the
modes, the element tables) give way, and the solve takes the stored K.

What a solve needs is counted on the same K as a tangent at zero displacement,
which has no such tables; a linear solve has to get by with that and with
every amount between that and all of its tables.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import openfea_b200 as ob
from openfea_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,shape,nrhs", [("GPU_MIXED", (40, 12, 11), 1), ("GPU_MIXED", (95, 36, 33), 1),
                                               ("GPU_LEARNED", (40, 12, 11), 1), ("GPU_PCG", (62, 35, 32), 1),
                                               ("GPU_MIXED", (40, 12, 11), 5)])
def test_optional_tables_give_way(gpu_ctx_factory, method, shape, nrhs):
    m = mg.structured_hex(*shape, *(0.005 * s for s in shape), 210e9, 0.3)
    f = K = None

    def context(linear=True):
        nonlocal f, K
        c = gpu_ctx_factory()
        c.upload_mesh(m)
        c.assemble_pattern()
        c.assemble_linear()
        if method == "GPU_LEARNED":
            c.learned_train(sample_iters=64, sample_every=4, steps=10, batch=8)
        if not linear:
            c.assemble_nl(np.zeros(c.n))
        if f is None:
            f = np.random.default_rng(7).normal(size=(c.n, nrhs))
            rp, col, val = c.get_csr()
            K = sp.csr_matrix((val, col, rp), shape=(c.n, c.n))
        return c

    def solve(c):
        u, st = c.solve(f if nrhs > 1 else f[:, 0], method=method, rtol=1e-8)
        u = u.reshape(c.n, nrhs)
        floor = np.diff(K.indptr).max() * np.finfo(float).eps * np.linalg.norm(abs(K) @ abs(u), axis=0)
        assert np.all(np.linalg.norm(f - K @ u, axis=0) <= 1e-8 * np.linalg.norm(f, axis=0) + floor)
        return u

    def taken(c):
        ob.limit_allocations()
        u = solve(c)
        return ob.limit_allocations(), u

    solve(context())  # every kernel loaded, the load-case shape tuned
    plain, _ = taken(context(linear=False))
    full, u_full = taken(context())
    assert full > plain
    for budget in (full - 1, (plain + full) // 2, plain):
        c = context()
        try:
            ob.limit_allocations(budget)
            solve(c)
        finally:
            ob.limit_allocations()
        solve(c)  # the tables stay away until the next pattern
        c.assemble_pattern()
        c.assemble_linear()
        again, u = taken(c)
        assert again > 0 and np.array_equal(u, u_full)
