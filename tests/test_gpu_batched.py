"""The persistent batched solver (ofea_batch_*): several SIMP design variants
of uneven length x several load cases, solved by one cooperative kernel,
against the per-variant solver, the oracle's assembly + a direct solve, its
own determinism, and the failure path of its grid barrier."""
import json
import os
import re

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

import openfea_b200 as ob
from openfea_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def variants(factory, count=4, nrhs=5, nmin=4, nmax=9):
    out = []
    for m, F in mg.design_variants(count=count, nrhs=nrhs, ny=4, nz=4, nmin=nmin, nmax=nmax):
        ctx = factory()
        fm = ctx.upload_mesh(m)
        ctx.assemble_pattern()
        ctx.assemble_linear()
        loads = np.stack([mg.to_free(F[j], fm) for j in range(nrhs)])
        out.append((ctx, m, fm, loads))
    return out


def true_rel_residual(ctx, U, F):
    rp, ci, val = ctx.get_csr()
    K = sp.csr_matrix((val, ci, rp), shape=(ctx.n, ctx.n))
    return max(np.linalg.norm(F[j] - K @ U[j]) / np.linalg.norm(F[j]) for j in range(F.shape[0]))


@pytest.mark.parametrize("method", ["GPU_MIXED", "GPU_PCG"])
def test_batched_matches_per_variant_solves(gpu_ctx_factory, tmp_path, monkeypatch, method):
    monkeypatch.setenv("OFEA_TUNE_FILE", str(tmp_path / "tune.json"))
    vs = variants(gpu_ctx_factory)
    b = ob.Batch([v[0] for v in vs], 5)
    U, st = b.solve([v[3] for v in vs], method=method, rtol=1e-10)
    for (ctx, m, fm, F), u, s in zip(vs, U, st):
        assert s["status"] == 0 and s["rel_residual"] <= 1e-10, s
        assert true_rel_residual(ctx, u, F) <= 1e-10
        ref, _ = ctx.solve(F.T, method="GPU_PCG", rtol=1e-13)
        assert np.linalg.norm(u - ref.T) / np.linalg.norm(ref) < 1e-8
    # the autotuner chose a configuration and kept it on disk
    t = b.tuning(method)
    assert t["rhs_per_lane"] in (1, 2, 4) and t["threads"] == 32 * 8 // t["rhs_per_lane"] and t["ms_per_iteration"] > 0
    data = json.load(open(tmp_path / "tune.json"))
    assert any("nrhs=5" in e["key"] for e in data["entries"])
    b.close()


def test_batched_against_oracle_direct_solve(gpu_ctx_factory, oracle):
    vs = variants(gpu_ctx_factory, count=2, nrhs=3)
    U, st = ob.solve_batched([v[0] for v in vs], [v[3] for v in vs], method="GPU_MIXED", rtol=1e-10)
    for (ctx, m, fm, F), u in zip(vs, U):
        cp, ri, val = oracle.assemble(m, fm)
        K = sp.csc_matrix((val, ri, cp), shape=(ctx.n, ctx.n))
        ref = spla.spsolve(K, F.T)
        assert np.linalg.norm(u - ref.T) / np.linalg.norm(ref) < 1e-8


# relative residual of the batched solves in the benchmark and here
BATCH_RTOL = 1e-8


@pytest.mark.parametrize("method", ["GPU_MIXED", "GPU_PCG"])
def test_batched_config4_variants_against_reference_superlu_class(gpu_ctx_factory, reference, method):
    """Real variants of the batched-reanalysis workload (64 SIMP variants
    n x 20 x 20, n ~ U{20..60}, 16 load cases): its three shortest variants
    (26,460-29,106 DOF), all 16 load cases, solved in one batch at the
    benchmark's residual, against the reference's reanalysis solver on its
    own K: solution_api("SuperLU_class") factors K and solves load case 0,
    superlu_solution_next re-solves the other 15 with that factor
    (src/linear_solution.cpp:23-39, src/solver/solver_superlu.cpp:76-94).
    Every load case within 1e-8 (relative L2)."""
    allv = mg.design_variants()
    pick = sorted(range(len(allv)), key=lambda i: (allv[i][0].nd, i))[:3]
    ctxs, loads, refs = [], [], []
    for i in pick:
        m, F = allv[i]
        ctx = gpu_ctx_factory()
        fm = ctx.upload_mesh(m)
        ctx.assemble_pattern()
        ctx.assemble_linear()
        Ff = np.stack([mg.to_free(F[j], fm) for j in range(F.shape[0])])
        rm = reference.model(m)
        rm.assemble()
        refs.append(rm.solve_multi(Ff))
        ctxs.append(ctx)
        loads.append(Ff)
    U, st = ob.solve_batched(ctxs, loads, method=method, rtol=BATCH_RTOL)
    worst = 0.0
    for u, ref, s in zip(U, refs, st):
        assert s["status"] == 0 and s["rel_residual"] <= BATCH_RTOL, s
        for j in range(ref.shape[0]):
            worst = max(worst, np.linalg.norm(u[j] - ref[j]) / np.linalg.norm(ref[j]))
    assert worst <= 1e-8, worst


def test_batched_is_deterministic_and_handles_one_load_case(gpu_ctx_factory):
    vs = variants(gpu_ctx_factory, count=3, nrhs=1)
    b = ob.Batch([v[0] for v in vs], 1)
    U1, _ = b.solve([v[3] for v in vs], method="GPU_MIXED", rtol=1e-9)
    U2, _ = b.solve([v[3] for v in vs], method="GPU_MIXED", rtol=1e-9)
    for a, c in zip(U1, U2):
        assert np.array_equal(a, c)
    b.close()


def test_batched_rejects_too_many_load_cases(gpu_ctx_factory):
    vs = variants(gpu_ctx_factory, count=1, nrhs=1)
    with pytest.raises(ob.OfeaError) as e:
        ob.Batch([vs[0][0]], 33)
    assert e.value.code == -7


def test_grid_barrier_wait_runs_out_and_context_stays_usable(gpu_ctx_factory):
    vs = variants(gpu_ctx_factory, count=1, nrhs=2)
    ctx = vs[0][0]
    assert ob.check_barrier_timeout(ctx, limit_ms=20) == 0
    b = ob.Batch([ctx], 2)
    U, st = b.solve([vs[0][3]], method="GPU_MIXED", rtol=1e-9)
    assert st[0]["status"] == 0
    b.close()


@pytest.mark.parametrize("method", ["GPU_MIXED", "GPU_PCG"])
@pytest.mark.parametrize("nrhs", [2, 17])
def test_copy_wait_runs_out_and_batch_stays_usable(gpu_ctx_factory, method, nrhs):
    # copies into shared memory that never complete: the kernels end with the
    # error, nothing of the copies is used, and the batch solves afterwards
    vs = variants(gpu_ctx_factory, count=3, nrhs=nrhs)
    b = ob.Batch([v[0] for v in vs], nrhs)
    before, _ = b.solve([v[3] for v in vs], method=method, rtol=1e-9)
    assert b.check_copy_timeout(method, limit_ms=20) == 0
    after, st = b.solve([v[3] for v in vs], method=method, rtol=1e-9)
    assert all(s["status"] == 0 for s in st)
    assert all(np.array_equal(x, y) for x, y in zip(before, after))
    b.close()


def test_batched_mixes_element_types(gpu_ctx_factory, oracle):
    """A batch holding a C3D4 tet block (per-element E) beside C3D8 variants:
    each variant is solved against its own K (checked with the oracle's)."""
    vs = variants(gpu_ctx_factory, count=2, nrhs=4)
    m, ffull = mg.tet_block(8, 4, 4)
    ctx = gpu_ctx_factory()
    fm = ctx.upload_mesh(m)
    ctx.assemble_pattern()
    ctx.assemble_linear()
    rng = np.random.default_rng(3)
    Ft = np.stack([mg.to_free(ffull * rng.uniform(0.5, 2.0), fm) for _ in range(4)])
    items = vs + [(ctx, m, fm, Ft)]
    U, st = ob.solve_batched([v[0] for v in items], [v[3] for v in items], method="GPU_MIXED", rtol=1e-10)
    for (c, mm, ff, F), u, s in zip(items, U, st):
        assert s["status"] == 0
        cp, ri, val = oracle.assemble(mm, ff)
        K = sp.csc_matrix((val, ri, cp), shape=(c.n, c.n))
        for j in range(F.shape[0]):
            assert np.linalg.norm(F[j] - K @ u[j]) <= 1.0001e-10 * np.linalg.norm(F[j])


@pytest.mark.parametrize("method,init,per_iter", [("GPU_MIXED", 8, 10), ("GPU_PCG", 4, 4)])
def test_batched_phase_trace(gpu_ctx_factory, tmp_path, monkeypatch, method, init, per_iter):
    # one launch: the init phases, then per iteration every phase but the
    # last iteration's V-cycle (the loop ends after the convergence check)
    monkeypatch.setenv("OFEA_TUNE_FILE", str(tmp_path / "tune.json"))
    vs = variants(gpu_ctx_factory, count=2, nrhs=3)
    b = ob.Batch([v[0] for v in vs], 3)
    with pytest.raises(ob.OfeaError):
        b.phase_times()  # tracing is off
    b.set_trace(100000)
    _, st = b.solve([v[3] for v in vs], method=method, rtol=1e-9)
    assert all(s["status"] == 0 and s["refinements"] == 0 for s in st), st
    it = max(s["iterations"] for s in st)
    t = b.phase_times()
    expect = init + per_iter * it if method == "GPU_PCG" else init + per_iter * (it - 1) + 4
    assert len(t) == expect
    assert np.all(t > 0) and t.sum() <= 1e3 * st[0]["seconds"]
    # a short trace keeps the first phases only
    b.set_trace(5)
    b.solve([v[3] for v in vs], method=method, rtol=1e-9)
    assert len(b.phase_times()) == 5
    b.set_trace(0)
    with pytest.raises(ob.OfeaError):
        b.phase_times()
    b.close()


def test_stored_tuning_is_for_its_kernels_and_matrices(gpu_ctx_factory, tmp_path, monkeypatch):
    # an entry of the file decides for the kernels, the preconditioner form and
    # the slices it was measured with, and for no others
    path = tmp_path / "tune.json"
    monkeypatch.setenv("OFEA_TUNE_FILE", str(path))

    def tuned(mesh, tangent=False):
        c = gpu_ctx_factory()
        c.upload_mesh(mesh)
        c.assemble_pattern()
        if tangent:
            c.assemble_nl(np.zeros(c.n))
        else:
            c.assemble_linear()
        b = ob.Batch([c], 4)
        t = b.tuning("GPU_MIXED")
        b.close()
        return t, {e["key"] for e in json.load(open(path))["entries"]}

    hexa = mg.structured_hex(9, 8, 5, 0.045, 0.04, 0.025, 210e9, 0.3)
    _, first = tuned(hexa)
    assert len(first) == 1
    (key,) = first
    _, again = tuned(hexa)
    assert again == first
    _, both = tuned(hexa, tangent=True)
    assert len(both) == 2 and first < both
    # what a build before this one wrote: device, method, load cases, rows, variants
    path.write_text('{"entries": [\n{"key": "%s", "rl": 1, "ctas_per_sm": 1, "ms_per_iter": 123.0}\n]}'
                    % "|".join(key.split("|")[:5]))
    t, keys = tuned(hexa)
    assert t["ms_per_iteration"] != 123.0 and key in keys


@pytest.mark.parametrize("method", ["GPU_MIXED", "GPU_PCG"])
@pytest.mark.parametrize("nrhs", [2, 5, 9, 17, 32])
def test_staged_and_direct_columns(gpu_ctx_factory, method, nrhs):
    # slices whose distinct columns fit the products' buffer and slices (many
    # load cases in FP64; a cross-section of 30 x 30 nodes) beyond it, every
    # load-case stride, C3D4 columns that are not in runs: the residual of
    # each load case on the host
    meshes = [mg.structured_hex(5, 2, 3, 0.025, 0.01, 0.015, 210e9, 0.3),
              mg.structured_hex(4, 29, 29, 0.02, 0.145, 0.145, 210e9, 0.3), mg.tet_block(5, 4, 3)[0]]
    ctxs, loads = [], []
    for i, m in enumerate(meshes):
        c = gpu_ctx_factory()
        c.upload_mesh(m)
        c.assemble_pattern()
        c.assemble_linear()
        ctxs.append(c)
        loads.append(np.random.default_rng(i).normal(size=(nrhs, c.n)))
    U, _ = ob.Batch(ctxs, nrhs).solve(loads, method=method, rtol=1e-9)
    for c, F, u in zip(ctxs, loads, U):
        rp, col, val = c.get_csr()
        K = sp.csr_matrix((val, col, rp), shape=(c.n, c.n))
        floor = np.diff(rp).max() * np.finfo(float).eps * np.linalg.norm(abs(K) @ abs(u.T), axis=0)
        norms = np.linalg.norm(F, axis=1)
        assert np.all(np.linalg.norm(F.T - K @ u.T, axis=0) <= 1e-9 * norms + floor)


@pytest.mark.parametrize("tangent", [False, True])
@pytest.mark.parametrize("nrhs", [1, 6, 20])
def test_vcycle_with_and_without_sparse_modes(gpu_ctx_factory, tangent, nrhs):
    # K Z exists for linear assemblies only: one variant with a tangent (at
    # zero displacement, the same K) sends the whole batch to the products.
    # Aggregates cut into more parts than some have K Z entries for.
    meshes = [mg.structured_hex(n, 6, 5, 0.05 * n, 0.3, 0.25, 210e9, 0.3) for n in (1, 9, 30)]
    ctxs, loads = [], []
    for i, m in enumerate(meshes):
        c = gpu_ctx_factory()
        c.upload_mesh(m)
        c.assemble_pattern()
        if tangent and i == 1:
            c.assemble_nl(np.zeros(c.n))
        else:
            c.assemble_linear()
        ctxs.append(c)
        loads.append(np.random.default_rng(i).normal(size=(nrhs, c.n)))
    U, _ = ob.Batch(ctxs, nrhs).solve(loads, method="GPU_MIXED", rtol=1e-9)
    for c, F, u in zip(ctxs, loads, U):
        rp, col, val = c.get_csr()
        K = sp.csr_matrix((val, col, rp), shape=(c.n, c.n))
        floor = np.diff(rp).max() * np.finfo(float).eps * np.linalg.norm(abs(K) @ abs(u.T), axis=0)
        norms = np.linalg.norm(F, axis=1)
        assert np.all(np.linalg.norm(F.T - K @ u.T, axis=0) <= 1e-9 * norms + floor)


@pytest.mark.parametrize("shape,nodes,kz_batch,kz_single", [((30, 12, 12), 1000, 1, True), ((30, 12, 12), 250, 1, True),
                                                            ((30, 12, 12), 30, 0, True), ((130, 25, 22), 30, 0, False)])
def test_sparse_modes_by_entries_per_row(gpu_ctx_factory, tmp_path, monkeypatch, shape, nodes, kz_batch, kz_single):
    # 0.4 to 4 entries of K Z per row: the batch takes it to 1.5, a single solve
    # to 8 (3.2 from 70,000 rows); a count that the batch did without is taken
    # again by the single solve
    path = tmp_path / "tune.json"
    monkeypatch.setenv("OFEA_TUNE_FILE", str(path))
    c = gpu_ctx_factory()
    c.upload_mesh(mg.structured_hex(*shape, *(0.005 * s for s in shape), 210e9, 0.3))
    c.assemble_pattern()
    c.set_coarse_nodes(nodes)
    c.assemble_linear()
    F = np.random.default_rng(5).normal(size=(3, c.n))
    b = ob.Batch([c], 3)
    (ub,), _ = b.solve([F], method="GPU_MIXED", rtol=1e-9)
    (key,) = {e["key"] for e in json.load(open(path))["entries"]}
    assert "kz=%d" % kz_batch in key
    c.set_setup_trace(True)
    us, _ = c.solve(F[0], method="GPU_MIXED", rtol=1e-9)
    if kz_batch == 0:  # else its values are there already
        assert ("modes" in c.setup_phase_times()) == kz_single
    rp, col, val = c.get_csr()
    K = sp.csr_matrix((val, col, rp), shape=(c.n, c.n))
    for u, f in [(us, F[0])] + list(zip(ub, F)):
        floor = np.diff(rp).max() * np.finfo(float).eps * np.linalg.norm(abs(K) @ abs(u))
        assert np.linalg.norm(f - K @ u) <= 1e-9 * np.linalg.norm(f) + floor
    (again,), _ = b.solve([F], method="GPU_MIXED", rtol=1e-9)
    assert np.array_equal(again, ub)
    b.close()


@pytest.mark.parametrize("nrhs", [3, 8, 16, 20, 32])
@pytest.mark.parametrize("rl", [1, 2, 4])
def test_every_tile_configuration(gpu_ctx_factory, tmp_path, monkeypatch, rl, nrhs):
    # whichever configuration the tuner finds fastest has to run: each by a
    # stored choice, every load-case stride and both methods
    path = tmp_path / "tune.json"
    monkeypatch.setenv("OFEA_TUNE_FILE", str(path))
    c = gpu_ctx_factory()
    c.upload_mesh(mg.structured_hex(5, 4, 3, 0.025, 0.02, 0.015, 210e9, 0.3))
    c.assemble_pattern()
    c.assemble_linear()
    rp, col, val = c.get_csr()
    K = sp.csr_matrix((val, col, rp), shape=(c.n, c.n))
    F = np.random.default_rng(nrhs).normal(size=(nrhs, c.n))
    for method in ("GPU_MIXED", "GPU_PCG"):
        b = ob.Batch([c], nrhs)
        b.tuning(method)
        b.close()
    stored = re.sub(r'"rl": \d+', '"rl": %d' % rl, path.read_text())
    path.write_text(re.sub(r'"ctas_per_sm": \d+', '"ctas_per_sm": 1', stored))  # one entry per line
    for method in ("GPU_MIXED", "GPU_PCG"):
        b = ob.Batch([c], nrhs)
        assert b.tuning(method)["rhs_per_lane"] == rl
        (u,), _ = b.solve([F], method=method, rtol=1e-9)
        floor = np.diff(rp).max() * np.finfo(float).eps * np.linalg.norm(abs(K) @ abs(u.T), axis=0)
        assert np.all(np.linalg.norm(F.T - K @ u.T, axis=0) <= 1e-9 * np.linalg.norm(F, axis=1) + floor)
        b.close()
