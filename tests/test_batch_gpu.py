"""Batched BiCGStab (one persistent, graph-captured launch) against the
single-system solver and against itself: every system converges, matches its
single-system solution, and is bitwise identical alone and in the mix."""
import numpy as np
import pytest
import scipy.sparse as sp

import block_matrix_format_performance_gb300 as bm

pytestmark = pytest.mark.gpu


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def q4_systems(grids):
    out = []
    for nx, ny in grids:
        rp, c, v, rhs = bm.gen_q4_elasticity(nx, ny)
        out.append((rp, c, v, rhs, 2))
    return out


def csr_of(rp, c, v, bs):
    crp, cc, cv = bm.bcsr_to_csr(rp, c, v, bs)
    return sp.csr_matrix((cv, cc, crp))


def run_batch(systems, precision="fp64", config=None, tol=1e-10, **kw):
    import torch
    mats = [bm.Matrix.from_bcsr(rp, c, v, bs) for rp, c, v, _, bs in systems]
    batch = bm.Batch(mats, precision, tol=tol, **kw)
    if config:
        batch.configure(*config)
    d_b = [dev(s[3]) for s in systems]
    d_x = [torch.full_like(b, float("nan")) for b in d_b]
    infos = batch.solve(d_b, d_x)
    xs = [x.cpu().numpy() for x in d_x]
    batch.close()
    for m in mats:
        m.close()
    return xs, infos


GRIDS = [(20, 5), (64, 16), (24, 6), (40, 10), (100, 25), (30, 8), (52, 13), (20, 5), (80, 20)]


@pytest.mark.parametrize("config", [(1, 256), (4, 256), (8, 512)])
def test_fp64_batch_converges_and_matches_single_solver(lib, cuda, config):
    systems = q4_systems(GRIDS)
    xs, infos = run_batch(systems, "fp64", config)
    misses = 0
    for (rp, c, v, rhs, bs), x, info in zip(systems, xs, infos):
        K = csr_of(rp, c, v, bs)
        rel = np.linalg.norm(rhs - K @ x) / np.linalg.norm(rhs)
        assert abs(rel - info["true_rel_residual"]) <= 1e-12 + 1e-3 * rel
        # Status must agree with the true residual; BiCGStab's path near the
        # FP64 accuracy of these operators depends on the team's summation
        # order, so one of the larger systems may end just above 1e-10.
        assert (info["status"] == bm.SUCCESS) == (rel < 1e-10), info
        if info["status"] != bm.SUCCESS:
            misses += 1
            assert rel < 3e-10 and len(rhs) >= 2 * 64 * 16, info
        A = bm.Matrix.from_bcsr(rp, c, v, bs)
        xs1, i1 = bm.Solver(A, "fp64").solve_host(rhs)
        assert np.linalg.norm(x - xs1) / np.linalg.norm(xs1) < 1e-7
    assert misses <= 1


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("config", [(1, 64), (2, 64), (8, 64), (1, 128), (2, 192), (8, 448), (1, 512)])
def test_every_team_shape_solves(lib, cuda, config, precision):
    """Teams with fewer warps than sums and than side-by-side divides (64
    threads), warp counts that are no power of two, one CTA and the largest
    cluster; systems smaller than a team and with rows left over. FP32 with a
    right-hand side at 1e-30: its dot products (1e-60) need FP64's range."""
    systems = []
    for nx, ny in ((2, 2), (20, 5), (33, 9), (64, 16)):
        rp, c, v, rhs = bm.gen_q4_elasticity(nx, ny)
        rows = np.repeat(np.arange(nx * ny), np.diff(rp))
        v.reshape(-1, 2, 2)[c == rows] += 0.05 * np.eye(2)
        rhs = np.random.default_rng(nx).uniform(-1, 1, rhs.size)
        systems.append((rp, c, v, rhs * (1e-30 if precision == "fp32" else 1.0), 2))
    tol = 1e-5 if precision == "fp32" else 1e-10
    xs, infos = run_batch(systems, precision, config, tol=tol)
    for (rp, c, v, rhs, bs), x, info in zip(systems, xs, infos):
        K = csr_of(rp, c, v, bs)
        rel = np.linalg.norm((rhs - K @ x) / np.linalg.norm(rhs))
        # FP32: the recursive residual meets the tolerance; the true one may
        # stand a rounding of x (2^-24 ||K|| ||x|| / ||b||, below 2e-5 here) above it
        assert rel < (tol if precision != "fp32" else 4e-5), (rel, info)
        if precision != "fp32":
            assert info["status"] == bm.SUCCESS, info


def test_result_is_bitwise_the_same_alone_and_in_the_mix(lib, cuda):
    systems = q4_systems(GRIDS)
    xs_mix, inf_mix = run_batch(systems, "fp64", (4, 256))
    for k in (0, 4, 7):
        xs_one, inf_one = run_batch([systems[k]], "fp64", (4, 256))
        assert inf_one[0]["iterations"] == inf_mix[k]["iterations"]
        assert np.array_equal(xs_one[0].view(np.uint64), xs_mix[k].view(np.uint64))


def test_autotuner_picks_a_valid_configuration(lib, cuda):
    import torch
    systems = q4_systems(GRIDS[:6])
    mats = [bm.Matrix.from_bcsr(rp, c, v, bs) for rp, c, v, _, bs in systems]
    batch = bm.Batch(mats, "fp64")
    d_b = [dev(s[3]) for s in systems]
    d_x = [torch.empty_like(b) for b in d_b]
    c, t = batch.autotune(d_b, d_x, probe_iterations=8)
    assert c in (1, 2, 4, 8) and t in (256, 512)
    infos = batch.solve(d_b, d_x)
    assert all(i["status"] == bm.SUCCESS for i in infos)


def diag_dominant(nbr, bs, seed):
    rng = np.random.default_rng(seed)
    rows = [np.unique(np.concatenate([[i], rng.integers(max(0, i - 10), min(nbr, i + 11), 6)])) for i in range(nbr)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    c = np.concatenate(rows).astype(np.int32)
    v = rng.uniform(-1, 1, c.size * bs * bs)
    for i in range(nbr):
        k = rp[i] + int(np.where(rows[i] == i)[0][0])
        v[k * bs * bs:(k + 1) * bs * bs].reshape(bs, bs)[...] += np.eye(bs) * (len(rows[i]) * bs * 1.5)
    b = rng.uniform(-1, 1, nbr * bs)
    return rp, c, v, b, bs


def test_mixed_batch_refines_well_conditioned_systems(lib, cuda):
    systems = [diag_dominant(n, 2, s) for s, n in enumerate((100, 800, 2500, 300))]
    xs, infos = run_batch(systems, "mixed", (2, 256))
    for (rp, c, v, b, bs), x, info in zip(systems, xs, infos):
        K = csr_of(rp, c, v, bs)
        assert info["status"] == bm.SUCCESS, info
        assert info["iterations_fp32"] == info["iterations"] > 0 and info["used_fp64_fallback"] == 0
        assert np.linalg.norm(b - K @ x) / np.linalg.norm(b) < 1e-10


def test_mixed_batch_falls_back_on_ill_conditioned_systems(lib, cuda):
    systems = q4_systems([(100, 25), (20, 5), (64, 16)])
    xs, infos = run_batch(systems, "mixed", (4, 256), max_iters=50000)
    xs64, infos64 = run_batch(systems, "fp64", (4, 256), max_iters=50000)
    fresh = 0
    for (rp, c, v, rhs, bs), x, info, x64, i64 in zip(systems, xs, infos, xs64, infos64):
        K = csr_of(rp, c, v, bs)
        rel = np.linalg.norm(rhs - K @ x) / np.linalg.norm(rhs)
        rel64 = np.linalg.norm(rhs - K @ x64) / np.linalg.norm(rhs)
        # Near FP64's accuracy on these operators a solve may end just above
        # 1e-10 (the FP64 batch solve as well); the status says so.
        assert (info["status"] == bm.SUCCESS) == (rel < 1e-10), info
        assert rel < 3e-10 and rel <= max(1e-10, 1.5 * rel64), (info, rel64)
        if info["used_fp64_fallback"] and info["iterations"] - info["iterations_fp32"] == i64["iterations"]:
            # FP32 steps that gained < 100x: the FP64 finish starts from x = 0
            # and is the FP64 solve, bit for bit.
            assert np.array_equal(x.view(np.uint64), x64.view(np.uint64))
            fresh += 1
    assert fresh >= 1


def test_fp32_batch(lib, cuda):
    systems = [diag_dominant(n, 2, s) for s, n in enumerate((200, 900))]
    xs, infos = run_batch(systems, "fp32", (1, 256), tol=1e-5)
    for (rp, c, v, b, bs), x, info in zip(systems, xs, infos):
        K = csr_of(rp, c, v, bs)
        assert info["status"] == bm.SUCCESS
        assert np.linalg.norm(b - K @ x) / np.linalg.norm(b) < 1e-4


def test_mixed_block_sizes_and_csr_systems(lib, cuda):
    import torch
    systems = [diag_dominant(300, 3, 1), diag_dominant(200, 2, 2), diag_dominant(150, 4, 3)]
    xs, infos = run_batch(systems, "fp64", (2, 256))
    for (rp, c, v, b, bs), x, info in zip(systems, xs, infos):
        assert info["status"] == bm.SUCCESS
        assert np.linalg.norm(b - csr_of(rp, c, v, bs) @ x) / np.linalg.norm(b) < 1e-10
    # CSR handles (bs = 0) take the CSR row routine
    rp, c, v, b, bs = diag_dominant(400, 2, 5)
    crp, cc, cv = bm.bcsr_to_csr(rp, c, v, bs)
    A = bm.Matrix.from_csr(crp, cc, cv, len(crp) - 1)
    batch = bm.Batch([A], "fp64")
    d_b, d_x = [dev(b)], [torch.empty(b.size, dtype=torch.float64, device="cuda")]
    info = batch.solve(d_b, d_x)[0]
    assert info["status"] == bm.SUCCESS
    assert np.linalg.norm(b - sp.csr_matrix((cv, cc, crp)) @ d_x[0].cpu().numpy()) / np.linalg.norm(b) < 1e-10


def test_inner_stall_window_keeps_results_and_cuts_fp32_work(lib, cuda):
    # FP32 inner solves cannot progress on the elasticity operator: a run that
    # has not halved its residual within the window is abandoned early. The
    # solves still reach the tolerance through the FP64 finish.
    systems = q4_systems([(100, 25), (64, 16), (40, 10)])
    _, infos0 = run_batch(systems, "mixed", (4, 256), max_iters=50000, inner_stall_iterations=0)
    xs, infos16 = run_batch(systems, "mixed", (4, 256), max_iters=50000, inner_stall_iterations=16)
    for (rp, c, v, rhs, bs), x, info in zip(systems, xs, infos16):
        K = csr_of(rp, c, v, bs)
        rel = np.linalg.norm(rhs - K @ x) / np.linalg.norm(rhs)
        assert (info["status"] == bm.SUCCESS) == (rel < 1e-10), info
        assert rel < 3e-10, info  # FP64's accuracy floor on this operator, as in the FP64 batch
    assert sum(i["iterations_fp32"] for i in infos16) <= sum(i["iterations_fp32"] for i in infos0)
    rp, c, v, _, bs = systems[0]
    m = bm.Matrix.from_bcsr(rp, c, v, bs)
    try:
        with pytest.raises(bm.BmfpError):
            bm.Batch([m], "mixed", inner_stall_iterations=-1)
    finally:
        m.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_grids_within_fp64_reach_converge_in_the_batch(lib, cuda, precision):
    """97x24, 150x38 and 240x60 of the uneven batch (FP64 rounding floors
    1.7e-11, 3.1e-11, 6.4e-11) end below 1e-10 in b - A x inside a batch:
    the team solver replaces its recursive residual by the true one near
    convergence (before, they stopped at 1.0-1.04e-10)."""
    systems = q4_systems([(97, 24), (150, 38), (240, 60), (40, 10)])
    xs, infos = run_batch(systems, precision, (4, 512), max_iters=100000)
    for (rp, c, v, rhs, bs), x, info in zip(systems, xs, infos):
        K = csr_of(rp, c, v, bs)
        rel = np.linalg.norm(rhs - K @ x) / np.linalg.norm(rhs)
        assert info["status"] == bm.SUCCESS and rel < 1e-10, (info, rel)
        if precision == "fp64" and len(rhs) > 2 * 40 * 10:
            assert info["replacements"] >= 1, info


def test_mixed_result_is_bitwise_the_same_alone_and_in_the_mix(lib, cuda):
    """Mixed precision in the batch: elasticity systems (FP32 steps fail,
    FP64 finish) and well-conditioned ones (FP32 refinements) give the same
    bits and counts alone and inside a mix."""
    systems = q4_systems(GRIDS[:5]) + [diag_dominant(500, 2, 7), diag_dominant(1200, 2, 8)]
    xs_mix, inf_mix = run_batch(systems, "mixed", (4, 256), max_iters=50000)
    for k in (0, 4, 5, 6):
        xs_one, inf_one = run_batch([systems[k]], "mixed", (4, 256), max_iters=50000)
        for key in ("iterations", "iterations_fp32", "refinements", "used_fp64_fallback", "status"):
            assert inf_one[0][key] == inf_mix[k][key], (k, key, inf_one[0], inf_mix[k])
        assert np.array_equal(xs_one[0].view(np.uint64), xs_mix[k].view(np.uint64)), k
    assert inf_mix[5]["iterations_fp32"] > 0 and inf_mix[5]["used_fp64_fallback"] == 0
