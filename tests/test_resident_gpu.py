"""Resident step form (csrc/resident.cu): LPs whose matrix, vectors and state
fit in the shared memory of one thread-block cluster.

The form does the operations of the other forms on every segment and element;
only the compensated norms are added in another order, with FP64 totals that
differ in the last bits.  One rounding of the FP32 step sizes may flip from
that (6e-8 relative), so that after 128 steps the points agree to 128 x 6e-8 <
1e-5 of their scale; after a solve both meet the tolerance at the same
optimum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sih():
    import sih_pdhg

    if not sih_pdhg.GpuSolver.is_cuda_available():
        pytest.fail("GPU test run without a CUDA device")
    return sih_pdhg


def _dense_row_lp(sih, m, n, seed):
    """One row over every column (longer than a warp's rows of entries), the rest with few."""
    rng = np.random.default_rng(seed)
    rows = np.concatenate([np.zeros(n, int), rng.integers(1, m, 3 * n)])
    cols = np.concatenate([np.arange(n), np.repeat(np.arange(n), 3)])
    A = sih.SparseMatrix.from_triplets(m, n, rows, cols, rng.standard_normal(4 * n))
    x0 = rng.uniform(0, 1, n)
    ax = A.mat_vec(x0)
    y0 = -np.abs(rng.standard_normal(m))
    c = A.mat_trans_vec(y0) + rng.uniform(0, 1, n)
    return sih.Problem.from_arrays(A, c, np.zeros(n), np.full(n, 2.0), np.full(m, -np.inf), ax + 0.1)


def _problem(sih, kind):
    from sih_pdhg.generators import mixed_bounds_lp, small_random_lp, zipf_lp

    if kind == "dense_row":
        return _dense_row_lp(sih, 120, 1500, 0)
    if kind == "every_bound":
        return mixed_bounds_lp(seed=2)
    if kind == "zipf":
        return zipf_lp(900, 2000, 16000, seed=1)
    m, n, k = kind
    return small_random_lp(m, n, k, 1)


# one block; two; a full portable cluster; 16 blocks; lengths at and past a batch and a lane group
KINDS = [(2, 3, 1), (33, 64, 1), (50, 120, 4), (200, 500, 8), (700, 1500, 9), (1999, 4999, 8), (2500, 6000, 11),
         (40, 45, 33), "every_bound", "dense_row", "zipf"]


@pytest.mark.parametrize("kind", KINDS, ids=str)
def test_steps_equal_the_kernel_per_phase_form(sih, kind):
    p = _problem(sih, kind)
    cfg = sih.GpuPdhgConfig(max_iterations=128, tol_primal=1e-12, tol_dual=1e-12, tol_gap=1e-12)
    a = sih.solve_gpu_mixed(p, cfg, persistent=0)
    b = sih.solve_gpu_mixed(p, cfg)
    assert a.simplex_iterations == b.simplex_iterations and a.restarts == b.restarts
    assert a.step_rejections == b.step_rejections
    for u, v in ((a.x, b.x), (a.row_duals, b.row_duals)):
        assert np.max(np.abs(u - v), initial=0.0) <= 1e-5 * max(1.0, np.max(np.abs(u), initial=0.0))
    assert b.kernel_launches < a.kernel_launches / 10  # the whole period is one launch


# too large for a cluster: over every SM, from barely (30k entries a side more
# than a cluster holds) to half of the SMs' shared memory, and one that does not fit (the older kernels)
GRID = [("uniform", 9000, 20000, 5), ("uniform", 4001, 30011, 7), ("zipf", 30000, 60000, 400000), ("refinery", 12),
        ("uniform", 90000, 150000, 10)]


@pytest.mark.parametrize("kind", GRID, ids=str)
def test_grid_form_steps_equal_the_kernel_per_phase_form(sih, kind):
    from sih_pdhg.generators import refinery_lp, small_random_lp, zipf_lp

    if kind[0] == "uniform":
        p = small_random_lp(*kind[1:], 2)
    else:
        p = refinery_lp(kind[1], 1) if kind[0] == "refinery" else zipf_lp(*kind[1:], 2)
    cfg = sih.GpuPdhgConfig(max_iterations=128, tol_primal=1e-12, tol_dual=1e-12, tol_gap=1e-12)
    for compensated in (0, 2):
        a = sih.solve_gpu_mixed(p, cfg, persistent=0, staged_kib=-1, compensated=compensated)
        b = sih.solve_gpu_mixed(p, cfg, compensated=compensated)
        assert a.simplex_iterations == b.simplex_iterations and a.restarts == b.restarts
        assert a.step_rejections == b.step_rejections
        for u, v in ((a.x, b.x), (a.row_duals, b.row_duals)):
            assert np.max(np.abs(u - v)) <= 1e-5 * max(1.0, np.max(np.abs(u)))


@pytest.mark.parametrize("compensated", [0, 2])
def test_solves_to_the_same_optimum(sih, compensated):
    p = _problem(sih, (300, 700, 6))
    cfg = sih.GpuPdhgConfig(max_iterations=200000)
    a = sih.solve_gpu_mixed(p, cfg, persistent=0, compensated=compensated)
    b = sih.solve_gpu_mixed(p, cfg, compensated=compensated)
    assert a.is_optimal() and b.is_optimal()
    assert max(b.rel_primal, b.rel_dual, b.rel_gap) <= 1e-4
    assert abs(a.primal_objective - b.primal_objective) <= 4e-4 * (1 + abs(a.primal_objective))


def test_batch_of_unequal_instances(sih):
    """Instances that need other cluster shares and stop at other evaluations,
    and the same batch with one that does not fit (every instance then runs in
    the other forms)."""
    from sih_pdhg.generators import refinery_lp

    ps = [_problem(sih, k) for k in ((200, 500, 8), (2, 3, 1), (1999, 4999, 8), "every_bound", (700, 1500, 9))]
    cfg = sih.GpuPdhgConfig(max_iterations=20000)
    for extra in ([], [refinery_lp(24, 1)]):
        a = sih.solve_batch(ps + extra, cfg, persistent=0, autotune=0)
        b = sih.solve_batch(ps + extra, cfg, autotune=0)
        for u, v in zip(a, b):
            assert u.status == v.status
            assert abs(u.primal_objective - v.primal_objective) <= 4e-4 * (1 + abs(u.primal_objective))


def test_run_again_and_warm_start(sih):
    p = _problem(sih, (700, 1500, 9))
    with sih.PdhgHandle(p, sih.GpuPdhgConfig(max_iterations=20000), algorithm=sih.ALGO_MIXED) as h:
        h.run()
        a = h.result(0)
        h.run()
        b = h.result(0)
        assert a.is_optimal() and np.array_equal(a.x, b.x) and a.simplex_iterations == b.simplex_iterations
        h.set_start(0, a.x, a.row_duals, a.final_primal_weight)
        h.run()
        c = h.result(0)
    assert c.is_optimal() and c.simplex_iterations <= 64


@pytest.mark.parametrize("kind", KINDS, ids=str)
@pytest.mark.parametrize("iterations", [7, 130, 425])
def test_plain_iterations_are_those_of_the_task_kernels(sih, kind, iterations):
    """The plain algorithm in the cluster (iterations and checks, several checks
    a launch, a shorter last block) against its kernels launched one by one: no
    sum enters the iterates but the segments', so they are the same bits."""
    p = _problem(sih, kind)
    cfg = sih.GpuPdhgConfig(max_iterations=iterations, tol_primal=1e-9, tol_dual=1e-9)
    a = sih.GpuSolver.solve_ex(p, cfg, use_graph=0)
    b = sih.solve_gpu_pdhg(p, cfg)
    assert a.simplex_iterations == b.simplex_iterations and a.status == b.status
    assert b.kernel_launches < a.kernel_launches / 10
    np.testing.assert_array_equal(a.row_duals, b.row_duals)
    np.testing.assert_array_equal(a.x, b.x)
    # the checks sum with the iteration's lanes: FP32 sums of at most 1,500 terms in another order
    assert abs(a.ref_primal - b.ref_primal) <= 1e-4 * (1e-3 + a.ref_primal)
    assert abs(a.ref_dual - b.ref_dual) <= 1e-4 * (1e-3 + a.ref_dual)


def test_plain_stops_at_the_same_check(sih):
    p = _problem(sih, (200, 500, 8))
    cfg = sih.GpuPdhgConfig(max_iterations=8000)
    a = sih.GpuSolver.solve_ex(p, cfg, use_graph=0)
    b = sih.solve_gpu_pdhg(p, cfg)
    assert a.is_optimal() and b.is_optimal()
    assert abs(a.simplex_iterations - b.simplex_iterations) <= cfg.check_frequency


def test_batch_takes_the_clusters_only_where_their_turns_are_short(sih):
    """One cluster size for the whole batch: a large LP among hundreds of small
    ones would give each of them 16 blocks and a step some forty turns; that batch
    steps over the task engine.  The small ones alone, and unequal ones in a few
    turns, stay resident."""
    from sih_pdhg.generators import small_random_lp

    small = [small_random_lp(60, 150, 5, s) for s in range(300)]
    mid = [small_random_lp(m, 5 * m // 2, 8, m) for m in range(200, 2000, 100)]
    cfg = sih.GpuPdhgConfig(max_iterations=20000)
    for ps, form in ((small + [small_random_lp(5000, 12000, 8, 7)], 0), (small, 1), (mid, 1)):
        with sih.PdhgHandle(ps, cfg, algorithm=sih.ALGO_MIXED, autotune=0) as h:
            assert h.launch_shape()["persistent"] == form
            h.run()
            assert all(h.result(b).is_optimal() for b in (0, len(ps) // 2, len(ps) - 1))


def test_tuner_times_the_resident_form_too(sih):
    """autotune = 1 on an LP that the SMs' shared memory holds: a step takes half
    of what the fastest kernels take, so the tuner keeps the resident form (a few
    launches, not three a step), the second time from its cache, with the same
    point as without it."""
    from sih_pdhg.generators import refinery_lp

    p = refinery_lp(168, 0)
    cfg = sih.GpuPdhgConfig(max_iterations=512, tol_primal=1e-12, tol_dual=1e-12, tol_gap=1e-12)
    a = sih.solve_gpu_mixed(p, cfg, autotune=0)
    for _ in range(2):
        b = sih.solve_gpu_mixed(p, cfg, autotune=1)
        assert b.kernel_launches == a.kernel_launches < 512
        np.testing.assert_array_equal(a.x, b.x)


@pytest.mark.parametrize("kind", GRID, ids=str)
def test_grid_form_runs_where_the_sms_hold_the_lp(sih, kind):
    """The LPs above really take the grid form: thirteen launches to start and one for
    up to four evaluation periods of 64 steps.  The last does not fit and takes three
    launches a step; it steps over packs like its baseline above, so here against
    the task engine (staged gathers ask for it)."""
    from sih_pdhg.generators import refinery_lp, small_random_lp, zipf_lp

    if kind[0] == "uniform":
        p = small_random_lp(*kind[1:], 2)
    else:
        p = refinery_lp(kind[1], 1) if kind[0] == "refinery" else zipf_lp(*kind[1:], 2)
    cfg = sih.GpuPdhgConfig(max_iterations=128, tol_primal=1e-12, tol_dual=1e-12, tol_gap=1e-12)
    b = sih.solve_gpu_mixed(p, cfg)
    if kind != GRID[-1]:
        assert b.kernel_launches == 14
        return
    assert b.kernel_launches > 3 * 128
    a = sih.solve_gpu_mixed(p, cfg, persistent=0, staged_kib=64)
    assert a.simplex_iterations == b.simplex_iterations and a.restarts == b.restarts
    for u, v in ((a.x, b.x), (a.row_duals, b.row_duals)):
        assert np.max(np.abs(u - v)) <= 1e-5 * max(1.0, np.max(np.abs(u)))


@pytest.mark.parametrize("compensated", [0, 2])
def test_single_lp_kernel_beyond_the_sms_shared_memory(sih, compensated):
    """persistent = 2 on an LP that no resident form holds (3.25M nonzeros, 39 MB
    of entries): k_solo_steps, one launch a period beside the evaluation's,
    against the kernels per phase."""
    from sih_pdhg.generators import small_random_lp

    p = small_random_lp(60000, 130000, 25, 3)
    cfg = sih.GpuPdhgConfig(max_iterations=128, tol_primal=1e-12, tol_dual=1e-12, tol_gap=1e-12)
    a = sih.solve_gpu_mixed(p, cfg, persistent=0, compensated=compensated)
    with sih.PdhgHandle(p, cfg, algorithm=sih.ALGO_MIXED, persistent=2, compensated=compensated) as h:
        assert h.launch_shape()["persistent"] == 2
        h.run()
        b = h.result(0)
    # thirteen launches to start, two periods of a launch and an evaluation of six
    assert b.kernel_launches == 27 and a.kernel_launches > 3 * 128
    assert a.simplex_iterations == b.simplex_iterations and a.restarts == b.restarts
    assert a.step_rejections == b.step_rejections
    for u, v in ((a.x, b.x), (a.row_duals, b.row_duals)):
        assert np.max(np.abs(u - v)) <= 1e-5 * max(1.0, np.max(np.abs(u)))


def test_batch_beyond_the_clusters_is_tuned(sih):
    """autotune = -1 on a batch with an instance that no cluster holds: the tuner
    times the kernels' shapes, and a second handle of the same shape reuses what
    it chose; the resident batches have nothing to tune."""
    from sih_pdhg.generators import small_random_lp

    ps = [small_random_lp(300, 700, 6, 0), small_random_lp(9000, 20000, 5, 1)]
    cfg = sih.GpuPdhgConfig(max_iterations=20000)
    shapes = []
    for _ in range(2):
        with sih.PdhgHandle(ps, cfg, algorithm=sih.ALGO_MIXED) as h:
            shapes.append(h.launch_shape())
            h.run()
            res = [h.result(b) for b in range(2)]
            assert all(r.is_optimal() for r in res)
            # not the resident form: seven launches a period at least
            assert res[0].kernel_launches >= 7 * (max(r.simplex_iterations for r in res) // 64)
    assert shapes[0]["tuned"] == 1 and shapes[0] == shapes[1]
    assert shapes[0]["row_lanes"] in (0, 1, 2, 4, 8) and shapes[0]["col_lanes"] in (0, 1, 2, 4, 8)
