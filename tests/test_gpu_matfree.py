"""Solves of large linear C3D8 models, whose outer products are formed from the
elements (matfree.cu) and not from the stored K.

The checks are on the assembled K (the arrays the oracle tests pin to the
reference): the residual of the returned u in FP64 on the host, for elements
in the usual order (each standing on the one before), in a random order (no
two of them linked), with numbered-about nodes and distorted elements.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import openfea_b200 as ob
from openfea_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def model(shape, order, seed=5):
    m = mg.structured_hex(*shape, *(0.005 * s for s in shape), 210e9, 0.3)
    rng = np.random.default_rng(seed)
    ext = 0.005 * np.array(shape)
    inside = np.all((m.xyz > 1e-9) & (m.xyz < ext - 1e-9), axis=1)
    m.xyz[inside] += rng.uniform(-0.0005, 0.0005, (int(inside.sum()), 3))
    m.E = 210e9 * mg.simp_density(shape, 3) ** 3
    if order != "lines":
        p = rng.permutation(m.ne)
        m.topo, m.E = m.topo[p], m.E[p]
    if order == "nodes":
        new = rng.permutation(m.nd)  # node i becomes new[i]
        xyz = np.empty_like(m.xyz)
        xyz[new] = m.xyz
        m.xyz, m.topo, m.fix = xyz, (new[m.topo - 1] + 1).astype(np.int32), np.sort(new[m.fix - 1] + 1).astype(np.int32)
    return m


def residual(ctx, f, u):
    rp, col, val = ctx.get_csr()
    K = sp.csr_matrix((val, col, rp), shape=(f.size, f.size))
    floor = int(np.diff(rp).max()) * np.finfo(float).eps * np.linalg.norm(abs(K) @ abs(u))
    return np.linalg.norm(f - K @ u) / np.linalg.norm(f), floor / np.linalg.norm(f)


# 70,000 block rows and more take the elements; MIXED beyond the resident solver
@pytest.mark.parametrize("method,shape,order", [
    ("GPU_PCG", (62, 35, 32), "lines"), ("GPU_PCG", (62, 35, 32), "elements"), ("GPU_PCG", (61, 34, 33), "nodes"),
    ("GPU_MIXED", (95, 36, 33), "lines"), ("GPU_MIXED", (95, 36, 33), "elements")])
def test_solves_from_the_elements(gpu_ctx_factory, method, shape, order):
    m = model(shape, order)
    ctx = gpu_ctx_factory()
    ctx.upload_mesh(m)
    ctx.assemble_pattern()
    ctx.assemble_linear()
    assert ctx.n >= 3 * 70000
    f = np.random.default_rng(7).normal(size=ctx.n)
    u, st = ctx.solve(f, method=method, rtol=1e-9)
    rel, floor = residual(ctx, f, u)
    assert rel <= 1e-9 + floor
    u2, _ = ctx.solve(f, method=method, rtol=1e-9)
    assert np.array_equal(u, u2)


def test_the_current_k_is_solved(gpu_ctx_factory):
    # new moduli, and a tangent that the linear elements do not give
    m = model((62, 35, 32), "lines")
    ctx = gpu_ctx_factory()
    ctx.upload_mesh(m)
    ctx.assemble_pattern()
    f = np.random.default_rng(8).normal(size=ctx.n)
    for step in ("linear", "moduli", "tangent"):
        if step == "moduli":
            ctx.set_modulus(np.linspace(50e9, 90e9, m.ne), 70e9)
        if step == "tangent":
            ctx.assemble_nl(np.random.default_rng(9).uniform(-5e-5, 5e-5, ctx.n))
        else:
            ctx.assemble_linear()
        u, _ = ctx.solve(f, method="GPU_PCG", rtol=1e-9)
        rel, floor = residual(ctx, f, u)
        assert rel <= 1e-9 + floor, step


def test_element_tables_are_built_for_the_solves_that_use_them(gpu_ctx_factory):
    # MIXED on the resident kernel reads the stored K; plain PCG of the same
    # model then builds the tables (24 FP64 forces per element among them)
    m = model((62, 35, 32), "lines")
    ctx = gpu_ctx_factory()
    ctx.upload_mesh(m)
    ctx.assemble_pattern()
    ctx.assemble_linear()
    f = np.random.default_rng(7).normal(size=ctx.n)
    ctx.solve(f, method="GPU_MIXED", rtol=1e-6)
    try:
        ob.limit_allocations()
        ctx.solve(f, method="GPU_PCG", rtol=1e-6)
        assert ob.limit_allocations() >= 192 * m.ne
        ctx.solve(f, method="GPU_PCG", rtol=1e-6)
        assert ob.limit_allocations() < 192 * m.ne
    finally:
        ob.limit_allocations()


def test_profiled_kernels_are_those_the_solve_launches(gpu_ctx_factory):
    # elements, K Z or the stored K by what the solve of this K takes; nothing
    # where the resident kernel runs the iterations
    def names(ctx, method):
        f = np.random.default_rng(7).normal(size=ctx.n)
        ctx.solve(f, method=method, rtol=1e-6)
        ks = ctx.profile_iteration(method, reps=3)
        assert all(k["ms"] > 0 for k in ks)
        u, _ = ctx.solve(f, method=method, rtol=1e-9)  # the vectors it timed on are scratch
        rel, floor = residual(ctx, f, u)
        assert rel <= 1e-9 + floor
        return [k["name"] for k in ks]

    ctx = gpu_ctx_factory()
    ctx.upload_mesh(model((95, 36, 33), "lines"))
    ctx.assemble_pattern()
    ctx.assemble_linear()
    assert names(ctx, "GPU_PCG") == ["k_hex_forces", "k_pcg64_A", "k_pcg64_B"]
    assert names(ctx, "GPU_MIXED") == ["k_hex_forces", "k_fcg_A", "k_fcg_B", "k_restrict_modes", "coarse solve", "k_fcg_post"]
    ctx.assemble_nl(np.zeros(ctx.n))
    assert names(ctx, "GPU_PCG") == []
    assert names(ctx, "GPU_MIXED") == ["k_fcg_A", "k_fcg_B", "k_vc_resid", "k_restrict", "coarse solve", "k_prolong",
                                       "k_fcg_post"]
    small = gpu_ctx_factory()
    small.upload_mesh(model((12, 8, 6), "lines"))
    small.assemble_pattern()
    small.assemble_linear()
    assert names(small, "GPU_MIXED") == []
    small.learned_train(sample_iters=64, sample_every=4, steps=10, batch=8)
    assert names(small, "GPU_LEARNED") == ["k_fcg_A", "k_fcg_B", "k_restrict_modes", "learned coarse solve", "k_fcg_post"]


def test_learned_solve_from_the_elements_and_from_the_stored_k(gpu_ctx_factory):
    # the learned stage on the same weights: outer products from the elements
    # (and K Z), and from K loaded as a matrix
    m = model((62, 35, 32), "lines")
    a, b = gpu_ctx_factory(), gpu_ctx_factory()
    fm = a.upload_mesh(m)
    a.assemble_pattern()
    a.assemble_linear()
    a.learned_train(sample_iters=64, sample_every=4, steps=10, batch=8)
    rp, col, val = a.get_csr()
    b.upload_csc(m.xyz, fm, rp, col, val)
    b.set_learned_weights(a.learned_weights())
    f = np.random.default_rng(7).normal(size=a.n)
    ua, sa = a.solve(f, method="GPU_LEARNED", rtol=1e-9)
    ub, sb = b.solve(f, method="GPU_LEARNED", rtol=1e-9)
    for u in (ua, ub):
        rel, floor = residual(a, f, u)
        assert rel <= 1e-9 + floor
    assert [k["name"] for k in a.profile_iteration("GPU_LEARNED", reps=2)][0] == "k_hex_forces"
    assert [k["name"] for k in b.profile_iteration("GPU_LEARNED", reps=2)][0] == "k_fcg_A"
    assert abs(sa["iterations"] - sb["iterations"]) <= max(3, 0.1 * sb["iterations"])
