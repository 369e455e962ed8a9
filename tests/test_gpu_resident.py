"""The resident solver (every iteration of a solve in one launch, resident.cu).

Slices of 32 rows are shared by several warps and CTAs own whole slices: the
sizes cover a single partial slice, one slice per CTA with many warps on it,
several slices per CTA and several rounds of slices.  Checked against the
assembled K on the host (the same arrays the oracle tests pin to the
reference): the residual of the returned u in FP64.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import openfea_b200 as ob
from openfea_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def host_residual(ctx, f, u):
    """||f - K u|| / ||f|| and the rounding of that product itself."""
    rp, col, val = ctx.get_csr()
    K = sp.csr_matrix((val, col, rp), shape=(f.size, f.size))
    per_row = int(np.diff(rp).max())
    floor = per_row * np.finfo(float).eps * np.linalg.norm(abs(K) @ abs(u))
    return np.linalg.norm(f - K @ u) / np.linalg.norm(f), floor / np.linalg.norm(f)


@pytest.mark.parametrize("method", ["GPU_PCG", "GPU_MIXED"])
@pytest.mark.parametrize("kind,shape", [("hex", (2, 1, 1)), ("hex", (9, 2, 3)), ("hex", (41, 9, 8)),
                                        ("hex", (70, 17, 16)), ("tet", (3, 2, 2)), ("tet", (33, 21, 11))])
def test_resident_solve_meets_its_residual(gpu_ctx_factory, method, kind, shape):
    if kind == "hex":
        m = mg.structured_hex(*shape, *(0.005 * s for s in shape), 210e9, 0.3)
        m.E = 210e9 * mg.simp_density(shape, 3) ** 3
    else:
        m = mg.tet_block(*shape)[0]
    ctx = gpu_ctx_factory()
    ctx.upload_mesh(m)
    ctx.assemble_pattern()
    ctx.assemble_linear()
    f = np.random.default_rng(7).normal(size=ctx.n)
    u, st = ctx.solve(f, method=method, rtol=1e-10)
    rel, floor = host_residual(ctx, f, u)
    assert rel <= 1e-10 + floor
    # polled every few iterations, and again: the same iterates
    u2, st2 = ctx.solve(f, method=method, rtol=1e-10, check_every=3)
    assert st2["iterations"] == st["iterations"] and np.array_equal(u, u2)


@pytest.mark.parametrize("kind,shape", [("hex", (9, 3, 3)), ("hex", (40, 12, 11)), ("tet", (7, 6, 5)), ("tet", (25, 16, 12))])
def test_preconditioner_with_and_without_its_mode_table(gpu_ctx_factory, kind, shape):
    # the linear stiffness of a mesh: the V-cycle takes K Z; the same K loaded as
    # a matrix: it restricts the residual.  The same solution, and about the
    # same preconditioner (their counts differ by the smoother's BF16 rounding)
    m = mg.structured_hex(*shape, *(0.005 * s for s in shape), 210e9, 0.3) if kind == "hex" else mg.tet_block(*shape)[0]
    if kind == "hex":
        m.E = 210e9 * mg.simp_density(shape, 4) ** 3
    a, b = gpu_ctx_factory(), gpu_ctx_factory()
    fm = a.upload_mesh(m)
    a.assemble_pattern()
    a.assemble_linear()
    rp, col, val = a.get_csr()
    b.upload_csc(m.xyz, fm, rp, col, val)
    f = np.random.default_rng(3).normal(size=a.n)
    ua, sa = a.solve(f, method="GPU_MIXED", rtol=1e-10)
    ub, sb = b.solve(f, method="GPU_MIXED", rtol=1e-10)
    for ctx, u in ((a, ua), (b, ub)):
        rel, floor = host_residual(ctx, f, u)
        assert rel <= 1e-10 + floor
    assert abs(sa["iterations"] - sb["iterations"]) <= max(3, 0.1 * sb["iterations"])


@pytest.mark.parametrize("method", ["GPU_MIXED", "GPU_LEARNED"])
def test_a_reset_rebuilds_the_mode_table(gpu_ctx_factory, method):
    # precond_reset: the next solve pays for the whole set-up, as after an assembly
    m = mg.structured_hex(40, 12, 11, 0.2, 0.06, 0.055, 210e9, 0.3)
    ctx = gpu_ctx_factory()
    ctx.upload_mesh(m)
    ctx.assemble_pattern()
    ctx.assemble_linear()
    if method == "GPU_LEARNED":
        ctx.learned_train(sample_iters=64, sample_every=4, steps=10, batch=8)
    f = np.random.default_rng(3).normal(size=ctx.n)
    ctx.set_setup_trace(True)

    def phases():
        u, _ = ctx.solve(f, method=method, rtol=1e-9)
        return u, [p for p in ctx.setup_phase_times()]

    u0, first = phases()
    assert "modes" in first
    u1, again = phases()
    assert "modes" not in again
    ctx.precond_reset()
    u2, reset = phases()
    ctx.assemble_linear()
    u3, assembled = phases()
    assert "modes" in assembled and reset == assembled
    assert all(np.array_equal(u0, u) for u in (u1, u2, u3))


@pytest.mark.parametrize("shape,nodes,tangent", [((50, 16, 16), 60, False), ((80, 20, 20), 160, False), ((80, 20, 20), 100, False),
                                                 ((100, 27, 25), 350, False), ((100, 27, 25), 350, True), ((100, 27, 25), 250, True)])
def test_coarse_levels_on_both_sides_of_the_resident_limit(gpu_ctx_factory, shape, nodes, tangent):
    # 1,248 to 1,728 coarse unknowns: the resident kernel takes 1,536 at most,
    # 1,250 where the products could be formed from the elements
    ctx = gpu_ctx_factory()
    m = mg.structured_hex(*shape, *(0.005 * s for s in shape), 210e9, 0.3)
    ctx.upload_mesh(m)
    ctx.assemble_pattern()
    ctx.set_coarse_nodes(nodes)
    if tangent:
        ctx.assemble_nl(np.zeros(ctx.n))
    else:
        ctx.assemble_linear()
    f = np.random.default_rng(7).normal(size=ctx.n)
    u, _ = ctx.solve(f, method="GPU_MIXED", rtol=1e-9)
    rel, floor = host_residual(ctx, f, u)
    assert rel <= 1e-9 + floor
    assert 1200 < ctx.coarse_apply()[0] < 1800
    u2, _ = ctx.solve(f, method="GPU_MIXED", rtol=1e-9)
    assert np.array_equal(u, u2)


@pytest.mark.parametrize("method", ["GPU_PCG", "GPU_MIXED"])
def test_barrier_wait_runs_out_and_context_stays_usable(gpu_ctx_factory, method):
    m = mg.structured_hex(41, 9, 8, 0.2, 0.045, 0.04, 210e9, 0.3)
    ctx = gpu_ctx_factory()
    ctx.upload_mesh(m)
    ctx.assemble_pattern()
    ctx.assemble_linear()
    f = np.random.default_rng(7).normal(size=ctx.n)
    u, _ = ctx.solve(f, method=method, rtol=1e-9)
    assert ob.check_resident_timeout(ctx, method, limit_ms=20) == 0
    again, _ = ctx.solve(f, method=method, rtol=1e-9)
    assert np.array_equal(u, again)


def test_time_budget_ends_a_resident_solve(gpu_ctx_factory):
    # a budget that is over at the first poll: one launch of a few iterations,
    # the residual of what it reached, and the same solve without one afterwards
    m = mg.structured_hex(41, 9, 8, 0.2, 0.045, 0.04, 210e9, 0.3)
    ctx = gpu_ctx_factory()
    ctx.upload_mesh(m)
    ctx.assemble_pattern()
    ctx.assemble_linear()
    f = np.random.default_rng(7).normal(size=ctx.n)
    for method in ("GPU_PCG", "GPU_MIXED"):
        u, full = ctx.solve(f, method=method, rtol=1e-10)
        part, st = ctx.solve(f, method=method, rtol=1e-10, time_budget_s=1e-9, raise_on_error=False)
        assert st["status"] != 0 and 0 < st["iterations"] < full["iterations"]
        rel, floor = host_residual(ctx, f, part)
        assert 1e-10 < rel and abs(rel - st["rel_residual"]) <= 1e-6 * rel + floor
        again, _ = ctx.solve(f, method=method, rtol=1e-10)
        assert np.array_equal(u, again)
