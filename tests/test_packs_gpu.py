"""Steps of one LP over packs of uniform segments (csrc/warp.cuh, spmv_packs)
against the task engine (staged_kib > 0 keeps it): the same sums per segment,
the compensated norms added in another order with FP64 totals that differ in
the last bits.  One rounding of the FP32 step sizes may flip from that (6e-8
relative): after 128 steps the points agree to 128 x 6e-8 < 1e-5 of their scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sih():
    import sih_pdhg

    if not sih_pdhg.GpuSolver.is_cuda_available():
        pytest.fail("GPU test run without a CUDA device")
    return sih_pdhg


def _lp(sih, m, lengths, seed):
    """Columns of the given lengths, rows drawn at random (a row drawn twice counts once)."""
    rng = np.random.default_rng(seed)
    lengths = rng.permutation(lengths)
    n = len(lengths)
    cols = np.repeat(np.arange(n), lengths)
    key = np.unique(cols * m + rng.integers(0, m, len(cols)))
    cols, rows = key // m, key % m
    A = sih.SparseMatrix.from_triplets(m, n, rows, cols, rng.standard_normal(len(key)))
    x0 = rng.uniform(0, 1, n)
    ax = A.mat_vec(x0)
    y0 = -np.abs(rng.standard_normal(m))
    c = A.mat_trans_vec(y0) + rng.uniform(0, 1, n)
    return sih.Problem.from_arrays(A, c, np.zeros(n), np.full(n, 2.0), np.full(m, -np.inf), ax + 0.1)


# a window holds 384 entries, a pack 32 segments, a batch 4 entries per lane
CASES = {
    "edges": (40001, [0] * 37 + [1] * 9001 + [2, 3, 4, 5, 7, 8, 9] * 3001 + [11, 12, 13] * 701 + [31, 32, 33] * 501
              + [127, 128, 129] * 90 + [383, 384, 385] * 7 + [767, 768, 769, 1500, 20011]),
    "fewer_packs_than_warps": (700, [1500] * 450 + [1] * 33),
    "nine_long_rows": (9, [27] * 31000),
    "short": (300007, [1] * 150001 + [2] * 100003 + [0] * 99),
}


@pytest.mark.parametrize("compensated", [0, 2])
@pytest.mark.parametrize("name", CASES)
def test_steps_equal_the_task_engine(sih, name, compensated):
    p = _lp(sih, *CASES[name], seed=4)
    assert len(p.A.csr_values()) >= 250000  # from here on one LP takes packs
    cfg = sih.GpuPdhgConfig(max_iterations=128, tol_primal=1e-12, tol_dual=1e-12, tol_gap=1e-12)
    a = sih.solve_gpu_mixed(p, cfg, persistent=0, staged_kib=1, compensated=compensated)
    b = sih.solve_gpu_mixed(p, cfg, persistent=0, compensated=compensated)
    assert a.simplex_iterations == b.simplex_iterations and a.restarts == b.restarts
    assert a.step_rejections == b.step_rejections
    for u, v in ((a.x, b.x), (a.row_duals, b.row_duals)):
        assert np.max(np.abs(u - v)) <= 1e-5 * max(1.0, np.max(np.abs(u)))
    with sih.PdhgHandle(p, cfg, algorithm=sih.ALGO_MIXED, persistent=0, compensated=compensated) as h:
        for _ in range(2):
            h.run()
            np.testing.assert_array_equal(h.result(0).x, b.x)
