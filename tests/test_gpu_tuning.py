"""PCG launch tuning on the GPU (``-m gpu``): every launch variant solves the same system.

The variants (SpMV unroll, CTA size, resident row-state layout, row split by
calibrated CTA speed, the single-reduction CG recurrence) change only the
summation order of the grid reductions, where row state lives or the rounding of
mathematically equal recurrences, so a substep agrees with the default
configuration to float32 round-off (relative 1e-5 on the velocity increment at a
tight tolerance), and repeated substeps of one configuration are bit-identical.
"""

import ctypes

import numpy as np
import pytest
import torch
from gpu_helpers import rel_l2, scene_pair, to_np

from newton_solver_fem_gb300 import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _cuda(cuda_device):
    yield


def setting(solver, key):
    v = ctypes.c_int64()
    _lib.check(_lib.load().fem_get_tuning(solver._handle, key, ctypes.byref(v)))
    return v.value


def substep(model, solver, sc):
    solver.reset()
    s0, s1 = model.state(), model.state()
    solver.refresh_tangent(s0.particle_q)
    solver.step(s0, s1, None, None, sc.dt)
    torch.cuda.synchronize()
    return to_np(solver.velocity_increment), to_np(s1.particle_q)


VARIANTS = [
    {_lib.FEM_TUNE_SPMV_UNROLL: 1},
    {_lib.FEM_TUNE_SPMV_UNROLL: 2},
    {_lib.FEM_TUNE_CTA_THREADS: 1024},
    {_lib.FEM_TUNE_CTA_THREADS: 512, _lib.FEM_TUNE_GRID_CAP: 7},
    {_lib.FEM_TUNE_RESIDENT_LAYOUT: 0},
    {_lib.FEM_TUNE_RESIDENT_LAYOUT: 2},
    {_lib.FEM_TUNE_BALANCE: 1},
    {_lib.FEM_TUNE_RESIDENT_LAYOUT: 2, _lib.FEM_TUNE_BALANCE: 1},
    {_lib.FEM_TUNE_SPLIT_HEADROOM: 10, _lib.FEM_TUNE_BALANCE: 1},
    {_lib.FEM_TUNE_TAIL_PREFETCH: 0},
    {_lib.FEM_TUNE_TAIL_PREFETCH: 100},
    {_lib.FEM_TUNE_COMPACT_COLUMNS: 0},
    {_lib.FEM_TUNE_COMPACT_COLUMNS: 1},
    {_lib.FEM_TUNE_COMPACT_COLUMNS: 2},
    {_lib.FEM_TUNE_COMPACT_COLUMNS: 2, _lib.FEM_TUNE_SPMV_UNROLL: 1},
    {_lib.FEM_TUNE_L2_RESIDENT_BYTES: 0},
    {_lib.FEM_TUNE_L2_RESIDENT_BYTES: 1 << 20, _lib.FEM_TUNE_COMPACT_COLUMNS: 2},
    {_lib.FEM_TUNE_CG_VARIANT: 1},
    {_lib.FEM_TUNE_CG_VARIANT: 1, _lib.FEM_TUNE_RESIDENT_LAYOUT: 0},
    {_lib.FEM_TUNE_CG_VARIANT: 1, _lib.FEM_TUNE_RESIDENT_LAYOUT: 2},
    {_lib.FEM_TUNE_CG_VARIANT: 1, _lib.FEM_TUNE_COMPACT_COLUMNS: 1, _lib.FEM_TUNE_SPMV_UNROLL: 2},
    {_lib.FEM_TUNE_CG_VARIANT: 1, _lib.FEM_TUNE_BALANCE: 1},
]


@pytest.mark.parametrize("variant", VARIANTS, ids=lambda v: "-".join(f"{k}={x}" for k, x in v.items()))
def test_launch_variants_solve_the_same_system(variant):
    sc = scenes.hex_block_64(n=24)
    model, solver, _ = scene_pair(sc, linear_solver_tolerance=1e-6, linear_solver_maxiter=400, with_oracle=False)
    dv_ref, q_ref = substep(model, solver, sc)
    lib = _lib.load()
    for key, value in variant.items():
        _lib.check(lib.fem_set_tuning(solver._handle, key, value))
    for key, value in variant.items():
        assert setting(solver, key) == value
    dv, q = substep(model, solver, sc)
    dv2, q2 = substep(model, solver, sc)
    np.testing.assert_array_equal(dv, dv2)  # deterministic within a configuration
    np.testing.assert_array_equal(q, q2)
    assert rel_l2(dv, dv_ref) < 1e-5
    assert np.isfinite(dv).all()


def test_calibrated_split_survives_topology_refresh_and_rejects_bad_values():
    sc = scenes.tet_jittered_48(n=10)
    model, solver, _ = scene_pair(sc, with_oracle=False)
    lib = _lib.load()
    _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_BALANCE, 1))
    for key, bad in ((_lib.FEM_TUNE_BALANCE, 2), (_lib.FEM_TUNE_RESIDENT_LAYOUT, 3),
                     (_lib.FEM_TUNE_SPLIT_HEADROOM, -1), (_lib.FEM_TUNE_SPLIT_HEADROOM, 51),
                     (_lib.FEM_TUNE_TAIL_PREFETCH, 101)):
        assert lib.fem_set_tuning(solver._handle, key, bad) == _lib.FEM_ERR_BAD_ARG
    solver.refresh_topology(model.particle_q)
    assert setting(solver, _lib.FEM_TUNE_BALANCE) == 1
    s0, s1 = model.state(), model.state()
    solver.step(s0, s1, None, None, sc.dt)
    assert torch.isfinite(s1.particle_q).all()


def test_automatic_residency_and_column_mode():
    """A matrix that fits in 60% of L2 is kept there whole and read with per-row offsets; one that
    streams (no resident bytes) reads the offsets its slices share once per slice."""
    sc = scenes.hex_block_64(n=12)
    model, solver, _ = scene_pair(sc, with_oracle=False)
    lib = _lib.load()
    nslices = -(-model.particle_count // 32)
    assert setting(solver, _lib.FEM_TUNE_L2_RESIDENT_BYTES) == -2
    assert setting(solver, _lib.FEM_TUNE_RESIDENT_SLICES) == nslices
    assert setting(solver, _lib.FEM_TUNE_COMPACT_COLUMNS) == 1
    _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_L2_RESIDENT_BYTES, 0))
    assert setting(solver, _lib.FEM_TUNE_RESIDENT_SLICES) == 0
    assert setting(solver, _lib.FEM_TUNE_COMPACT_COLUMNS) == 2
    assert setting(solver, _lib.FEM_TUNE_UNIFORM_COLUMN_BLOCKS) > 0
    for key, bad in ((_lib.FEM_TUNE_L2_RESIDENT_BYTES, -3), (_lib.FEM_TUNE_COMPACT_COLUMNS, -2)):
        assert lib.fem_set_tuning(solver._handle, key, bad) == _lib.FEM_ERR_BAD_ARG


@pytest.mark.parametrize("cap,state", [(9, 1), (6, 0), (3, 0)])  # 55, 82 and 163 slices per CTA
@pytest.mark.parametrize("l2_bytes,depth", [(-2, 4), (0, 2)])
def test_automatic_depth_and_row_state_change_no_bit(cap, state, l2_bytes, depth):
    """A matrix that streams is read two blocks at a time, one that stays in L2 four; row state is kept in
    shared memory up to 160 KB unless it is asked for.  Neither changes the order of a sum."""
    sc = scenes.hex_block_64(n=24)
    model, solver, _ = scene_pair(sc, linear_solver_tolerance=1e-6, linear_solver_maxiter=100, with_oracle=False)
    lib = _lib.load()
    for key, value in ((_lib.FEM_TUNE_CTA_THREADS, 1024), (_lib.FEM_TUNE_GRID_CAP, cap),
                       (_lib.FEM_TUNE_L2_RESIDENT_BYTES, l2_bytes)):
        _lib.check(lib.fem_set_tuning(solver._handle, key, value))
    assert setting(solver, _lib.FEM_TUNE_SPMV_UNROLL) == depth
    assert setting(solver, _lib.FEM_TUNE_RESIDENT_STATE) == state
    got = substep(model, solver, sc)
    for key, value in ((_lib.FEM_TUNE_SPMV_UNROLL, 6 - depth), (_lib.FEM_TUNE_RESIDENT_LAYOUT, 1)):
        _lib.check(lib.fem_set_tuning(solver._handle, key, value))
    assert setting(solver, _lib.FEM_TUNE_SPMV_UNROLL) == 6 - depth
    assert setting(solver, _lib.FEM_TUNE_RESIDENT_STATE) == (1 if cap > 3 else 0)
    asked = substep(model, solver, sc)
    for a, b in zip(got, asked):
        np.testing.assert_array_equal(a, b)


def test_load_depth_is_saved_restored_and_reset():
    """Writing back the depth that was read, or the former default of 4, leaves the kernel and every bit of a
    substep as they are; 0 is automatic again."""
    sc = scenes.hex_block_64(n=12)
    model, solver, _ = scene_pair(sc, linear_solver_tolerance=1e-6, linear_solver_maxiter=100, with_oracle=False)
    lib = _lib.load()
    put = lambda key, value: _lib.check(lib.fem_set_tuning(solver._handle, key, value))  # noqa: E731
    for onchip in (-1, 0):
        put(_lib.FEM_TUNE_ONCHIP, onchip)
        put(_lib.FEM_TUNE_SPMV_UNROLL, 0)
        grid, ref = setting(solver, _lib.FEM_TUNE_ONCHIP_GRID), substep(model, solver, sc)
        assert (grid > 0) == (onchip == -1)
        for depth in (setting(solver, _lib.FEM_TUNE_SPMV_UNROLL), 4, 2, 1, 0):
            put(_lib.FEM_TUNE_SPMV_UNROLL, depth)
            assert setting(solver, _lib.FEM_TUNE_SPMV_UNROLL) == (depth or 4)
            assert setting(solver, _lib.FEM_TUNE_ONCHIP_GRID) == grid
            for a, b in zip(substep(model, solver, sc), ref):
                np.testing.assert_array_equal(a, b)
    put(_lib.FEM_TUNE_L2_RESIDENT_BYTES, 0)
    for depth, used in ((0, 2), (4, 4), (0, 2)):
        put(_lib.FEM_TUNE_SPMV_UNROLL, depth)
        assert setting(solver, _lib.FEM_TUNE_SPMV_UNROLL) == used
    for bad in (-1, 3, 8):
        assert lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_SPMV_UNROLL, bad) == _lib.FEM_ERR_BAD_ARG


def test_column_modes_are_bit_identical_and_report_shared_slots():
    """Column modes only change where a block's column comes from, so substeps agree bit for bit."""
    sc = scenes.hex_block_64(n=12)
    model, solver, _ = scene_pair(sc, with_oracle=False)
    lib = _lib.load()
    _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_COMPACT_COLUMNS, 2))
    assert setting(solver, _lib.FEM_TUNE_COMPACT_COLUMNS) == 2
    shared = setting(solver, _lib.FEM_TUNE_UNIFORM_COLUMN_BLOCKS)
    assert 0 < shared < solver.matrix_info()["nnzb"]
    ref = substep(model, solver, sc)
    for mode in (1, 0):
        _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_COMPACT_COLUMNS, mode))
        assert setting(solver, _lib.FEM_TUNE_UNIFORM_COLUMN_BLOCKS) == 0
        got = substep(model, solver, sc)
        np.testing.assert_array_equal(got[0], ref[0])
        np.testing.assert_array_equal(got[1], ref[1])
    assert lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_COMPACT_COLUMNS, 3) == _lib.FEM_ERR_BAD_ARG


def test_calibrated_split_of_a_spread_batch():
    """A 24-scene batch (slices dealt to CTAs in interleaved runs) re-split by calibrated CTA speed
    solves the same system, deterministically."""
    sc = scenes.batched_scenes(count=24, seed=5, dims=(3, 10))
    model, solver, _ = scene_pair(sc, linear_solver_tolerance=1e-6, linear_solver_maxiter=200, with_oracle=False)
    dv_ref, _ = substep(model, solver, sc)
    lib = _lib.load()
    _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_BALANCE, 1))
    dv, _ = substep(model, solver, sc)
    dv2, _ = substep(model, solver, sc)
    np.testing.assert_array_equal(dv, dv2)
    assert rel_l2(dv, dv_ref) < 1e-5


def test_handles_needing_different_pcg_shared_memory_launch_in_any_order():
    """Two systems of 32 and 24 slices each run as one CTA (a warp per slice), whose PCG launches need
    about 79 KB and 60 KB of dynamic shared memory, above the default 48 KB.  That limit belongs to the
    kernel, not the handle; configuring the smaller system after the larger must leave the larger one's
    cooperative launch (eager and graph-captured) valid, and every step must match a fresh handle."""
    from gpu_helpers import make_pair

    def pair(cells):
        x, hexes, mats, mass = scenes.hex_block(*cells, 0.05, (0.0, 0.0, 0.0), 1e5, 0.3, 1000.0)
        return make_pair(x, mass, hexes=hexes, hex_materials=mats, gravity=(0.0, 0.0, -9.81), with_oracle=False,
                         linear_solver_maxiter=40, linear_solver_tolerance=1e-6)

    big_model, big, _ = pair((9, 9, 9))      # 1,000 nodes: 32 slices
    small_model, small, _ = pair((7, 7, 11))  # 768 nodes: 24 slices
    assert setting(big, _lib.FEM_TUNE_GRID) == 1 and setting(big, _lib.FEM_TUNE_CTA_THREADS) == 1024
    assert setting(small, _lib.FEM_TUNE_GRID) == 1 and setting(small, _lib.FEM_TUNE_CTA_THREADS) == 768

    def run(model, solver, steps=3):
        s0, s1 = model.state(), model.state()
        solver.reset()
        solver.refresh_tangent(s0.particle_q)
        for _ in range(steps):
            solver.step(s0, s1, None, None, 1.0 / 600.0)
            s0, s1 = s1, s0
        torch.cuda.synchronize()
        return to_np(s0.particle_q)

    q_big, q_small = run(big_model, big), run(small_model, small)
    again_model, again, _ = pair((9, 9, 9))
    assert np.array_equal(run(again_model, again), q_big)
    assert np.array_equal(run(big_model, big), q_big)  # after the small handle was configured
    assert np.array_equal(run(small_model, small), q_small)

    s0, s1 = big_model.state(), big_model.state()
    big.reset()
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        big.refresh_tangent(s0.particle_q)
        big.step(s0, s1, None, None, 1.0 / 600.0)  # allocations outside capture
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            big.step(s0, s1, None, None, 1.0 / 600.0)
    pair((7, 7, 11))  # a third handle configured between capture and replay
    graph.replay()
    torch.cuda.synchronize()
    assert np.isfinite(to_np(s1.particle_q)).all()


# Slice and launch-shape edges of the on-chip kernel: one partial slice, exactly one and just over one
# slice (32 and 33 rows are not grid sizes; 27 and 36 straddle them), one CTA, a cluster, a grid with
# whole and with partly resident rows, and rows enough for the wide variant.
ONCHIP_SHAPES = [("hex", (1, 1, 1)), ("tet", (2, 2, 2)), ("hex", (3, 2, 2)), ("tet", (4, 4, 4)), ("hex", (5, 5, 4)),
                 ("tet", (4, 4, 16)), ("hex", (9, 9, 9)), ("hex", (13, 12, 11)), ("tet", (17, 13, 11)),
                 ("hex", (23, 17, 11)), ("hex", (33, 32, 31)), ("tet", (46, 43, 41)), ("hex", (43, 42, 41))]


@pytest.mark.parametrize("element,cells", ONCHIP_SHAPES, ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_onchip_kernel_solves_the_streaming_kernels_system(element, cells):
    """Same tight-tolerance substep from a deformed, moving start and a warm start, with a fixed face; the
    bound is the launch variants' one, as the recurrences agree to float32 round-off.  The adjoint-style
    solve from zero is held to the same bound, and repeated substeps are bit-identical."""
    from gpu_helpers import make_pair

    block = scenes.tet_block if element == "tet" else scenes.hex_block
    x, el, mats, mass = block(*cells, 0.01, (0.0, 0.0, 0.0), 2e5, 0.4, 1000.0)
    fixed = np.nonzero(np.isclose(x[:, 0], 0.0))[0].astype(np.int32)
    elements = {"tets": el, "tet_materials": mats} if element == "tet" else {"hexes": el, "hex_materials": mats}
    model, solver, _ = make_pair(x, mass, fixed=fixed, gravity=(0.0, 0.0, -9.81), with_oracle=False,
                                 linear_solver_tolerance=1e-6, linear_solver_maxiter=200, **elements)
    lib = _lib.load()
    rng = np.random.default_rng(31)
    q = torch.tensor((x + rng.normal(0.0, 2e-4, x.shape)).astype(np.float32), device="cuda")
    v = torch.tensor(rng.normal(0.0, 0.05, x.shape).astype(np.float32), device="cuda")
    warm = torch.tensor(rng.normal(0.0, 5e-3, x.shape).astype(np.float32), device="cuda")
    rhs = torch.tensor((rng.normal(0.0, 1.0, x.shape) * mass[:, None]).astype(np.float32), device="cuda")

    def run():
        s0, s1 = model.state(), model.state()
        s0.particle_q.copy_(q)
        s0.particle_qd.copy_(v)
        solver.refresh_tangent(s0.particle_q)
        solver.velocity_increment.copy_(warm)
        solver.step(s0, s1, None, None, 1.0 / 600.0)
        y = torch.empty_like(rhs)
        _lib.check(lib.fem_solve(solver._handle, rhs.data_ptr(), y.data_ptr(), 1e-6, 200, solver._stream()))
        torch.cuda.synchronize()
        assert solver.stats()["status"] == 0
        return to_np(solver.velocity_increment), to_np(s1.particle_q), to_np(y)

    assert setting(solver, _lib.FEM_TUNE_ONCHIP_GRID) > 0
    got, again = run(), run()
    _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_ONCHIP, 0))
    assert setting(solver, _lib.FEM_TUNE_ONCHIP_GRID) == 0
    ref = run()
    for a, b, c in zip(got, again, ref):
        np.testing.assert_array_equal(a, b)
        assert rel_l2(a, c) < 1e-5


@pytest.mark.parametrize("layers,ctas", [(8, 5), (9, 6), (11, 7), (14, 9), (16, 10), (17, 11), (20, 13), (22, 14), (24, 15)])
def test_onchip_clusters_of_any_size_solve_the_streaming_kernels_system(layers, ctas):
    """Clusters whose size is no multiple of four, where the lanes that hand totals to the peers make unequal
    numbers of trips before the cluster barrier: the launch variants' bound, and the same bits each time."""
    from gpu_helpers import make_pair

    x, hexes, mats, mass = scenes.hex_block(layers - 1, 4, 3, 0.01, (0.0, 0.0, 0.0), 2e5, 0.4, 1000.0)
    order = np.random.default_rng(0).permutation(len(x))  # every slice holds a row of 27 blocks: past the one-CTA limit
    x[order], mass[order], hexes = x.copy(), mass.copy(), order[hexes].astype(np.int32)
    fixed = np.nonzero(np.isclose(x[:, 0], 0.0))[0].astype(np.int32)
    model, solver, _ = make_pair(x, mass, fixed=fixed, hexes=hexes, hex_materials=mats, with_oracle=False,
                                 linear_solver_tolerance=1e-6, linear_solver_maxiter=200)
    lib = _lib.load()
    rhs = torch.tensor((np.random.default_rng(37).normal(0.0, 1.0, x.shape) * mass[:, None]).astype(np.float32),
                       device="cuda")

    def run():
        y = torch.empty_like(rhs)
        _lib.check(lib.fem_solve(solver._handle, rhs.data_ptr(), y.data_ptr(), 1e-6, 200, solver._stream()))
        torch.cuda.synchronize()
        assert solver.stats()["status"] == 0
        return to_np(y)

    assert setting(solver, _lib.FEM_TUNE_ONCHIP_GRID) == ctas
    got, again = run(), run()
    _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_ONCHIP, 0))
    np.testing.assert_array_equal(got, again)
    assert rel_l2(got, run()) < 1e-5


@pytest.mark.parametrize("element,cells", [("hex", (1, 1, 1)), ("tet", (1, 1, 1)), ("hex", (2, 2, 2)), ("hex", (3, 2, 2)),
                                           ("hex", (3, 3, 3)), ("tet", (40, 1, 1))])
def test_onchip_iterates_of_the_smallest_bodies_are_as_exact_as_the_streaming_kernels(element, cells):
    """Bodies that one CTA solves converge in steep last steps, where rounding in CG's scalars shows most.  After
    the steps that 64-bit CG takes to 1e-4, the mean distance from its iterates over 24 right-hand sides is at
    most half again the streaming kernel's (the same sums in another order, so samples of one spread)."""
    from gpu_helpers import make_pair

    block = scenes.tet_block if element == "tet" else scenes.hex_block
    x, el, mats, mass = block(*cells, 0.01, (0.0, 0.0, 0.0), 3e5, 0.4, 1000.0)
    fixed = np.nonzero(np.isclose(x[:, 0], 0.0))[0].astype(np.int32)
    elements = {"tets": el, "tet_materials": mats} if element == "tet" else {"hexes": el, "hex_materials": mats}
    model, solver, _ = make_pair(x, mass, fixed=fixed, with_oracle=False, **elements)
    P, lib = len(x), _lib.load()
    keep = np.ones((P, 3))
    keep[fixed] = 0.0
    keep = keep.ravel()
    A, minv = solver.A_bsr.dense().astype(np.float64), to_np(solver._pc_inv_diag).reshape(P, 3, 3)
    precondition = lambda r: np.einsum("nij,nj->ni", minv, r.reshape(P, 3)).ravel()  # noqa: E731
    off = {0: [], -1: []}
    for seed in range(24):
        b = (np.random.default_rng(seed).normal(0.0, 1.0, x.shape) * mass[:, None]).astype(np.float32)
        b[fixed] = 0.0
        rhs = torch.tensor(b, device="cuda")
        r = b.astype(np.float64).ravel()
        want, z, stop, steps = np.zeros(3 * P), precondition(r), 1e-8 * (r @ r), 0
        p, rz = z, r @ z
        while r @ r > stop:
            y = keep * (A @ p)
            alpha = rz / (p @ y)
            want, r = want + alpha * p, r - alpha * y
            z = precondition(r)
            p, rz = z + (r @ z) / rz * p, r @ z
            steps += 1
        for onchip in (0, -1):
            _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_ONCHIP, onchip))
            y = torch.empty_like(rhs)
            _lib.check(lib.fem_solve(solver._handle, rhs.data_ptr(), y.data_ptr(), 1e-30, steps, solver._stream()))
            off[onchip].append(rel_l2(to_np(y), want))
    assert np.mean(off[-1]) < 1.5 * np.mean(off[0])


@pytest.mark.parametrize("tolerance,maxiter", [(0.3, 50), (1e-4, 1)])  # ends by the threshold, and by the cap
@pytest.mark.parametrize("cells", [(9, 9, 9), (16, 15, 14)])  # a cluster, a grid
def test_onchip_reports_the_residual_after_a_steep_last_step(cells, tolerance, maxiter):
    """A right-hand side that is a generalised eigenvector of A and the preconditioner plus a fifth of noise: one
    step cuts ||r||^2 to 1 to 10 percent.  The reported residual is the 64-bit ||b - A x|| / ||b|| up to the rounding
    of a float sum, on the mean of 16 noises less than one float32 unit; a prediction is off by the cancelled factor."""
    sp = pytest.importorskip("scipy.sparse")
    from gpu_helpers import make_pair
    from scipy.sparse.linalg import eigsh

    x, hexes, mats, mass = scenes.hex_block(*cells, 0.01, (0.0, 0.0, 0.0), 2e5, 0.4, 1000.0)
    model, solver, _ = make_pair(x, mass, hexes=hexes, hex_materials=mats, with_oracle=False)
    P, bsr = len(x), solver.A_bsr
    at = (bsr.columns.cpu().numpy(), bsr.offsets.cpu().numpy())
    A = sp.bsr_matrix((to_np(bsr.values), *at), shape=(3 * P, 3 * P)).tocsr()
    minv = to_np(solver._pc_inv_diag).reshape(P, 3, 3)
    rows = (np.arange(P), np.arange(P + 1))
    M = sp.bsr_matrix((np.linalg.inv(minv), *rows), shape=A.shape).tocsc()
    v = eigsh(A, k=1, M=M, Minv=sp.bsr_matrix((minv, *rows), shape=A.shape).tocsc(), which="LM", v0=np.ones(3 * P))[1][:, 0]
    assert setting(solver, _lib.FEM_TUNE_ONCHIP_GRID) > 1
    off = []
    for seed in range(16):
        b, noise = A @ v, (np.random.default_rng(seed).normal(0.0, 1.0, x.shape) * mass[:, None]).ravel()
        b = (b / np.linalg.norm(b) + 0.2 * noise / np.linalg.norm(noise)).astype(np.float32)
        rhs = torch.tensor(b.reshape(P, 3), device="cuda")
        y = torch.empty_like(rhs)
        _lib.check(_lib.load().fem_solve(solver._handle, rhs.data_ptr(), y.data_ptr(), tolerance, maxiter, solver._stream()))
        b, got = b.astype(np.float64), solver.stats()
        true = np.linalg.norm(b - A @ to_np(y).ravel()) / np.linalg.norm(b)
        assert got["max_iterations"] == 1 and 0.1 < true < 0.33
        assert got["unconverged_scenes"] == (maxiter == 1)
        off.append(abs(got["max_relative_residual"] / true - 1.0))
    assert np.mean(off) < 2.0 ** -23


@pytest.mark.parametrize("element,cells,spread,onchip", [
    ("hex", (48, 48, 48), 0, True), ("hex", (51, 51, 51), 0, False), ("tet", (52, 52, 52), 0, True),
    ("tet", (34, 34, 34), -1, True), ("tet", (38, 38, 38), -1, False), ("hex", (33, 33, 33), -1, False),
    ("tet", (46, 46, 46), 300, True), ("tet", (46, 46, 46), 10000, False)])
def test_onchip_is_left_where_the_streaming_kernel_is_faster(element, cells, spread, onchip):
    """Large bodies whose columns do not stay in L2 and numberings without locality (a spread of -1 is random)
    stream by default; asked for, the on-chip kernel still solves the same system to the variants' bound."""
    from gpu_helpers import make_pair

    block = scenes.tet_block if element == "tet" else scenes.hex_block
    x, el, mats, mass = block(*cells, 0.01, (0.0, 0.0, 0.0), 2e5, 0.4, 1000.0)
    P, rng = len(x), np.random.default_rng(1)
    order = np.arange(P) if spread == 0 else np.argsort(np.arange(P) + rng.normal(0.0, spread if spread > 0 else 100.0 * P, P))
    place = np.empty(P, np.int64)
    place[order] = np.arange(P)
    x, mass, el = x[order], mass[order], place[el].astype(np.int32)
    elements = {"tets": el, "tet_materials": mats} if element == "tet" else {"hexes": el, "hex_materials": mats}
    model, solver, _ = make_pair(x, mass, with_oracle=False, **elements)
    lib = _lib.load()
    rhs = torch.tensor((rng.normal(0.0, 1.0, x.shape) * mass[:, None]).astype(np.float32), device="cuda")

    def solve(mode):
        _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_ONCHIP, mode))
        y = torch.empty_like(rhs)
        _lib.check(lib.fem_solve(solver._handle, rhs.data_ptr(), y.data_ptr(), 1e-6, 200, solver._stream()))
        assert solver.stats()["status"] == 0
        return to_np(y), setting(solver, _lib.FEM_TUNE_ONCHIP_GRID) > 0

    (auto, used), (asked, forced), (streamed, off) = solve(-1), solve(1), solve(0)
    assert used == onchip and forced and not off
    np.testing.assert_array_equal(auto, asked if onchip else streamed)
    assert rel_l2(asked, streamed) < 1e-5


@pytest.mark.parametrize("neighbours", [13856, 13917, 13918, 13919, 13920, 13921])
def test_hub_whose_halo_takes_all_shared_memory(neighbours):
    """A node joined to 13,856 others by springs leaves its CTA's shared memory no room for a block; from
    there to 13,921 the halo is within what an SM has but not within what a launch may ask for.  All are
    created and solved (by the streaming kernel where the halo does not fit); the star's solution is explicit."""
    from gpu_helpers import make_pair, tensor

    rng = np.random.default_rng(11)
    P, m, ke, kd, h = 32 + neighbours, 0.5, np.float32(40.0), np.float32(0.01), np.float64(np.float32(1.0 / 600.0))
    x = rng.uniform(0.0, 1.0, (P, 3))
    springs = np.stack([np.zeros(neighbours, np.int32), np.arange(32, P, dtype=np.int32)], 1)  # 1..31 stay free
    model, solver, _ = make_pair(x, np.full(P, m), springs=springs, spring_ke=np.full(neighbours, ke),
                                 spring_kd=np.full(neighbours, kd), with_oracle=False)
    rhs = tensor(rng.normal(0.0, 1.0, (P, 3)))
    y = torch.empty_like(rhs)
    _lib.check(_lib.load().fem_solve(solver._handle, rhs.data_ptr(), y.data_ptr(), 1e-6, 100, solver._stream()))
    assert solver.stats()["status"] == 0
    b, c = to_np(rhs), h * h * ke + h * kd
    want = b / m
    want[0] = (b[0] + c * b[32:].sum(0) / (m + c)) / (m + c * neighbours - neighbours * c * c / (m + c))
    want[32:] = (b[32:] + c * want[0]) / (m + c)
    assert rel_l2(to_np(y), want) < 1e-5


@pytest.mark.parametrize("count,dims", [(2, (2, 3)), (24, (3, 10)), (9, (2, 24)), (152, (2, 5))],
                         ids=lambda v: str(v).replace(" ", ""))
def test_onchip_teams_solve_the_streaming_kernels_batch(count, dims):
    """Scenes of one to many slices as teams of one to many CTAs, up to a scene per SM: the launch
    variants' bound against the streaming kernel, and repeated substeps are bit-identical."""
    sc = scenes.batched_scenes(count=count, seed=7, dims=dims)
    model, solver, _ = scene_pair(sc, linear_solver_tolerance=1e-6, linear_solver_maxiter=200, with_oracle=False)
    lib = _lib.load()
    assert setting(solver, _lib.FEM_TUNE_ONCHIP_GRID) >= count
    got, again = substep(model, solver, sc), substep(model, solver, sc)
    its = solver.stats()["scene_iterations"]
    _lib.check(lib.fem_set_tuning(solver._handle, _lib.FEM_TUNE_ONCHIP, 0))
    ref = substep(model, solver, sc)
    assert max(abs(a - b) for a, b in zip(its, solver.stats()["scene_iterations"])) <= 1
    for a, b, c in zip(got, again, ref):
        np.testing.assert_array_equal(a, b)
        assert rel_l2(a, c) < 1e-5
