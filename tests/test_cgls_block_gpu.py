"""CGLS with a block per instance (csrc/adjoint.cu, k_cgls_block) against the
kernels of a batch with an instance that does not fit a block.  Both refine in
FP64 to a residual of 1e-9 or less; bases of these LPs have condition numbers up
to about 1e4, so gradients and vertices agree to 1e-5 of their scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sih():
    import sih_pdhg

    if not sih_pdhg.GpuSolver.is_cuda_available():
        pytest.fail("GPU test run without a CUDA device")
    return sih_pdhg


def _large(sih, n=9000):
    """min -sum x, x <= 1 by rows of the identity: 9,000 rows and columns, more than a block holds."""
    A = sih.SparseMatrix.from_triplets(n, n, np.arange(n), np.arange(n), np.ones(n))
    p = sih.Problem.from_arrays(A, -np.ones(n), np.zeros(n), np.full(n, 2.0), np.full(n, -np.inf), np.ones(n))
    return p, np.ones(n), np.ones(n)


# rows of 133 entries (more than 4 x 32); a few entries; near the limit of a block (10,800 nonzeros)
SHAPES = [(3, 5, 3, 0), (50, 120, 4, 1), (60, 400, 20, 0), (200, 500, 8, 0), (300, 1200, 9, 0)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_block_form_equals_the_kernels(sih, shape):
    from sih_pdhg.generators import small_random_lp

    p = small_random_lp(*shape)
    cfg = sih.GpuPdhgConfig(max_iterations=1_000_000, tol_primal=1e-6, tol_dual=1e-6, tol_gap=1e-6)
    s = sih.solve_gpu_mixed(p, cfg)
    q, xq, yq = _large(sih)
    g = np.random.default_rng(5).standard_normal(p.num_cols())
    ga, ia = sih.adjoint_batch([p], [s.x], [s.row_duals], [g])
    gb, ib = sih.adjoint_batch([p, q], [s.x, xq], [s.row_duals, yq], [g, np.ones(9000)])
    assert ia[0]["status"] == ib[0]["status"] == 0
    assert max(ia[0]["residual"], ib[0]["residual"]) <= 1e-9
    assert abs(ia[0]["iterations"] - ib[0]["iterations"]) <= 0.1 * ib[0]["iterations"] + 2
    for k in ("row_lower", "row_upper", "col_lower", "col_upper"):
        scale = max(1.0, np.abs(gb[0][k]).max())
        np.testing.assert_allclose(ga[0][k], gb[0][k], rtol=0, atol=1e-5 * scale)
    xa, ya, ja = sih.polish_batch([p], [s.x], [s.row_duals])
    xb, yb, jb = sih.polish_batch([p, q], [s.x, xq], [s.row_duals, yq])
    assert ja[0]["status"] == jb[0]["status"] == 0
    np.testing.assert_allclose(xa[0], xb[0], rtol=0, atol=1e-5 * max(1.0, np.abs(xb[0]).max()))
    np.testing.assert_allclose(ya[0], yb[0], rtol=0, atol=1e-5 * max(1.0, np.abs(yb[0]).max()))


def test_block_form_stops_at_the_iteration_limit(sih):
    from sih_pdhg.generators import small_random_lp

    p = small_random_lp(100, 250, 6, 0)
    rng = np.random.default_rng(0)
    x, y = rng.uniform(0, 1, 250), rng.standard_normal(100)
    _, info = sih.adjoint_batch([p, p], [x, x], [y, y], [np.ones(250)] * 2, max_iterations=3)
    for i in info:
        assert i["status"] == 1 and i["iterations"] == 12  # three in each of four rounds


def test_threads_with_batches_of_different_sizes(sih):
    """Entry points are re-entrant: calls on batches near a block's limit and on
    small ones at the same time (every launch asks for its own amount of shared
    memory) succeed and return what they return alone."""
    import threading

    from sih_pdhg.generators import small_random_lp

    def call(p):
        r = np.random.default_rng(3)
        x, y = r.uniform(0, 1, p.num_cols()), r.standard_normal(p.num_rows())
        g, info = sih.adjoint_batch([p, p], [x, x], [y, y], [np.ones(p.num_cols())] * 2, max_iterations=50)
        return np.concatenate([np.concatenate([q[k] for k in sorted(q)]) for q in g])

    ps = [small_random_lp(300, 1200, 9, 0), small_random_lp(50, 120, 4, 0)]
    alone = [call(p) for p in ps]
    wrong = []

    def work(i):
        for _ in range(40):
            try:
                if not np.array_equal(call(ps[i]), alone[i]):
                    wrong.append("other results")
            except sih._lib.SihPdhgError as e:
                wrong.append(str(e))

    threads = [threading.Thread(target=work, args=(i % 2,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]
