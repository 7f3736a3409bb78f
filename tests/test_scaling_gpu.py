"""Set-up scaling passes (csrc/mixed.cu, k_scale_pass) where their split of a side
changes: empty segments, groups of one lane and of more, segments around and past
the 256 entries from which a whole warp takes them.  Against the FP64 oracle after
16 steps: FP32 rounding of sums of up to 700 terms and 32 products is below 1e-3 of
the point's scale, a segment scaled wrongly moves its entries by its own size."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sih():
    import sih_pdhg

    if not sih_pdhg.GpuSolver.is_cuda_available():
        pytest.fail("GPU test run without a CUDA device")
    return sih_pdhg


@pytest.mark.parametrize("side", ["columns", "rows"])
@pytest.mark.parametrize("short, long", [([0, 1, 2, 3, 5, 7, 8], [255, 256, 257, 289, 700]), ([40] * 7, [300, 513])])
@pytest.mark.parametrize("passes", [(10, 1), (1, 0), (0, 1), (0, 0)])
def test_scaled_steps_follow_the_oracle(sih, side, short, long, passes):
    rng = np.random.default_rng(7)
    nseg, other = 700, 20011  # so many on the other side that its segments stay short
    lengths = rng.permutation(np.array(long + short * ((nseg - len(long)) // len(short))))
    seg = np.repeat(np.arange(len(lengths)), lengths)
    key = np.unique(seg * other + rng.integers(0, other, len(seg)))
    seg, idx = key // other, key % other
    m, n = (other, len(lengths)) if side == "columns" else (len(lengths), other)
    rows, cols = (idx, seg) if side == "columns" else (seg, idx)
    vals = rng.standard_normal(len(key)) * 10.0 ** rng.uniform(-1, 1, len(key))
    A = sih.SparseMatrix.from_triplets(m, n, rows, cols, vals)
    ax = A.mat_vec(rng.uniform(0, 1, n))
    c = A.mat_trans_vec(-np.abs(rng.standard_normal(m))) + rng.uniform(0, 1, n)
    p = sih.Problem.from_arrays(A, c, np.zeros(n), np.full(n, 2.0), np.full(m, -np.inf), ax + 0.1)
    cfg = sih.GpuPdhgConfig(max_iterations=16, tol_primal=1e-12, tol_dual=1e-12, tol_gap=1e-12)
    opts = dict(eval_frequency=16, ruiz_iterations=passes[0], pock_chambolle=passes[1])
    s = sih.solve_gpu_mixed(p, cfg, compensated=2, **opts)
    x, y, info = oracle.pdlp_solve(p, max_attempts=16, tol=1e-12, **opts)
    assert s.step_rejections == info["rejections"]
    assert np.max(np.abs(s.x - x)) <= 1e-3 * np.max(np.abs(x))
    assert np.max(np.abs(s.row_duals - y)) <= 1e-3 * np.max(np.abs(y))
