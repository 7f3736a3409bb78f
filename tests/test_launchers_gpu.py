"""The reference-compatible launchers (include/sih_pdhg.h sih_pdhg_launch_*)
against the oracle's restatement of core/src/gpu/cuda_pdhg.cu kernels.
SpMVs: FP32 tolerance (different summation order); elementwise kernels:
bit for bit (same unfused float operations)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    import oracle
    import sih_pdhg
    from sih_pdhg import _lib

    if not torch.cuda.is_available():
        pytest.fail("GPU test run without a CUDA device")
    return torch, _lib.load(), oracle


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("shape", [(2000, 5000, 8), (300, 700, 40), (50, 60, 1)])
def test_spmv_launchers(env, shape):
    torch, lib, oracle = env
    from sih_pdhg.generators import small_random_lp

    m, n, k = shape
    p = small_random_lp(m, n, k, 4)
    A = p.A
    rp, ci, rv = A.csr_row_ptr().astype(np.int32), A.csr_col_ind().astype(np.int32), A.csr_values().astype(np.float32)
    cp, ri, cv = A.csc_col_ptr().astype(np.int32), A.csc_row_ind().astype(np.int32), A.csc_values().astype(np.float32)
    rng = np.random.default_rng(1)
    x = rng.standard_normal(n).astype(np.float32)
    y = rng.standard_normal(m).astype(np.float32)
    d = {k2: _dev(torch, v) for k2, v in dict(rp=rp, ci=ci, rv=rv, cp=cp, ri=ri, cv=cv, x=x, y=y).items()}
    ax = torch.zeros(m, dtype=torch.float32, device="cuda")
    aty = torch.zeros(n, dtype=torch.float32, device="cuda")
    assert lib.sih_pdhg_launch_csr_spmv(m, d["rp"].data_ptr(), d["ci"].data_ptr(), d["rv"].data_ptr(),
                                        d["x"].data_ptr(), ax.data_ptr(), None) == 0
    assert lib.sih_pdhg_launch_csc_spmv(n, d["cp"].data_ptr(), d["ri"].data_ptr(), d["cv"].data_ptr(),
                                        d["y"].data_ptr(), aty.data_ptr(), None) == 0
    torch.cuda.synchronize()
    ref_ax = oracle.csr_spmv_f32(rp, ci, rv, x)
    ref_aty = oracle.csc_spmv_f32(cp, ri, cv, y)
    # FP32 sums of k terms: |error| <= k * eps * sum |a_i x_i|
    abs_ax = np.bincount(np.repeat(np.arange(m), np.diff(rp)), weights=np.abs(rv * x[ci]), minlength=m)
    abs_aty = np.bincount(np.repeat(np.arange(n), np.diff(cp)), weights=np.abs(cv * y[ri]), minlength=n)
    tol_ax = 2 * max(1, np.diff(rp).max()) * 1.2e-7 * abs_ax + 1e-30
    tol_aty = 2 * max(1, np.diff(cp).max()) * 1.2e-7 * abs_aty + 1e-30
    assert np.all(np.abs(ax.cpu().numpy() - ref_ax) <= tol_ax)
    assert np.all(np.abs(aty.cpu().numpy() - ref_aty) <= tol_aty)


def test_update_launchers_bit_exact(env):
    torch, lib, oracle = env
    rng = np.random.default_rng(2)
    n, m = 10_001, 7_003
    tau = rng.uniform(0.01, 1, n).astype(np.float32)
    c = rng.standard_normal(n).astype(np.float32)
    aty = rng.standard_normal(n).astype(np.float32)
    l = np.where(rng.random(n) < 0.1, -np.inf, rng.uniform(-1, 0, n)).astype(np.float32)
    u = np.where(rng.random(n) < 0.1, np.inf, rng.uniform(0, 2, n)).astype(np.float32)
    x = rng.uniform(-1, 1, n).astype(np.float32)
    sig = rng.uniform(0.01, 1, m).astype(np.float32)
    axb = rng.standard_normal(m).astype(np.float32)
    rl = np.where(rng.random(m) < 0.5, -np.inf, rng.uniform(-1, 0, m)).astype(np.float32)
    ru = np.where(rng.random(m) < 0.3, np.inf, rng.uniform(0, 1, m)).astype(np.float32)
    ru[:100] = rl[:100] = 0.25  # equality rows
    y = rng.standard_normal(m).astype(np.float32)
    d = {k: _dev(torch, v) for k, v in dict(tau=tau, c=c, aty=aty, l=l, u=u, x=x, sig=sig, axb=axb, rl=rl, ru=ru,
                                               y=y).items()}
    xbar = torch.zeros(n, dtype=torch.float32, device="cuda")
    assert lib.sih_pdhg_launch_primal_update(n, d["tau"].data_ptr(), d["c"].data_ptr(), d["aty"].data_ptr(),
                                             d["l"].data_ptr(), d["u"].data_ptr(), d["x"].data_ptr(),
                                             xbar.data_ptr(), None) == 0
    assert lib.sih_pdhg_launch_dual_update(m, d["sig"].data_ptr(), d["axb"].data_ptr(), d["rl"].data_ptr(),
                                           d["ru"].data_ptr(), d["y"].data_ptr(), None) == 0
    rv = torch.zeros(m, dtype=torch.float32, device="cuda")
    cvl = torch.zeros(n, dtype=torch.float32, device="cuda")
    assert lib.sih_pdhg_launch_residuals(m, n, d["axb"].data_ptr(), d["rl"].data_ptr(), d["ru"].data_ptr(),
                                         rv.data_ptr(), d["x"].data_ptr(), d["c"].data_ptr(), d["aty"].data_ptr(),
                                         d["l"].data_ptr(), d["u"].data_ptr(), d["tau"].data_ptr(),
                                         cvl.data_ptr(), None) == 0
    xb2 = torch.zeros(n, dtype=torch.float32, device="cuda")
    assert lib.sih_pdhg_launch_restart(n, d["x"].data_ptr(), xb2.data_ptr(), None) == 0
    torch.cuda.synchronize()
    x_ref, xbar_ref = oracle.primal_update_f32(tau, c, aty, l, u, x)
    y_ref = oracle.dual_update_f32(sig, axb, rl, ru, y)
    np.testing.assert_array_equal(d["x"].cpu().numpy(), x_ref)
    np.testing.assert_array_equal(xbar.cpu().numpy(), xbar_ref)
    np.testing.assert_array_equal(d["y"].cpu().numpy(), y_ref)
    np.testing.assert_array_equal(xb2.cpu().numpy(), x_ref)
    # residual maps (cuda_pdhg.cu:114-151) recomputed in numpy float32
    a = axb
    viol = np.zeros(m, np.float32)
    lo = (rl > -1e15) & (a < rl)
    viol[lo] = (rl - a)[lo]
    hi = (ru < 1e15) & (a > ru)
    viol[hi] = np.maximum(viol[hi], (a - ru)[hi])
    np.testing.assert_array_equal(rv.cpu().numpy(), viol)
    xn = x_ref
    proj = (xn - tau * (c + aty)).astype(np.float32)
    proj = np.minimum(np.maximum(proj, l), u)
    meas = (np.abs(xn - proj) / np.maximum(np.float32(1e-4), tau)).astype(np.float32)
    np.testing.assert_array_equal(cvl.cpu().numpy(), meas)


@pytest.mark.parametrize("nseg", [1, 31, 32767, 32768, 32769, 40001])
@pytest.mark.parametrize("kind", ["mixed", "short", "long"])
def test_spmv_launcher_by_segment_count_and_lengths(env, nseg, kind):
    """Both ways of the SpMV kernel (groups of lanes; from 32,768 segments and
    below a mean of 64 entries, 32 segments a warp by stream) on empty
    segments and lengths around a lane's, a warp's and a window's share.  FP32
    products and sums of k terms: |error| <= (k + 1) eps sum |a x|."""
    torch, lib, _ = env
    rng = np.random.default_rng(nseg)
    lens = {"mixed": rng.choice([0, 1, 2, 7, 31, 32, 33, 48, 49, 255], nseg),
            "short": rng.integers(0, 4, nseg), "long": np.full(nseg, 70)}[kind]
    for k, v in ((3, 513), (nseg // 2, 2047), (nseg - 1, 512)):  # windows end inside and at segments
        if k < nseg and kind != "long":
            lens[k] = v
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    nnz, nvec = int(ptr[-1]), 5000
    idx = rng.integers(0, nvec, nnz).astype(np.int32)
    val = rng.standard_normal(nnz).astype(np.float32)
    vec = rng.standard_normal(nvec).astype(np.float32)
    d = [_dev(torch, a) for a in (ptr, idx, val, vec)]
    out = torch.full((nseg,), 7.0, dtype=torch.float32, device="cuda")
    for fn in (lib.sih_pdhg_launch_csr_spmv, lib.sih_pdhg_launch_csc_spmv):
        out.fill_(7.0)
        assert fn(nseg, *[a.data_ptr() for a in d], out.data_ptr(), None) == 0
        torch.cuda.synchronize()
        seg = np.repeat(np.arange(nseg), lens)
        prod = val.astype(np.float64) * vec[idx]
        ref = np.bincount(seg, weights=prod, minlength=nseg)
        tol = (lens + 1) * 1.2e-7 * np.bincount(seg, weights=np.abs(prod), minlength=nseg)
        assert np.all(np.abs(out.cpu().numpy() - ref) <= tol + 1e-30)


def test_chained_launchers_see_each_other(env):
    """Launchers wait on the device for the kernel before them: a chain in one
    stream, each reading what the one before wrote, and a copy behind it."""
    torch, lib, _ = env
    n = 200_000
    s = torch.cuda.Stream()
    a = torch.zeros(n, device="cuda")
    b = torch.zeros(n, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for k in range(1, 21):
            a.add_(1.0)  # not a chained kernel
            assert lib.sih_pdhg_launch_restart(n, a.data_ptr(), b.data_ptr(), s.cuda_stream) == 0
            assert lib.sih_pdhg_launch_restart(n, b.data_ptr(), a.data_ptr(), s.cuda_stream) == 0
            assert float(b.min()) == k and float(a.max()) == k


def _spmv(torch, lib, lens, idx, val, vec):
    nseg = len(lens)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    d = [_dev(torch, a) for a in (ptr, idx.astype(np.int32), val, vec)]
    out = torch.full((nseg,), 7.0, dtype=torch.float32, device="cuda")
    assert lib.sih_pdhg_launch_csr_spmv(nseg, *[a.data_ptr() for a in d], out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("length", [3, 20, 31, "uneven"])
def test_spmv_by_stream_loses_only_the_products_roundings(env, length):
    """40,000 short segments go by stream (a mean below 32, asserted): products
    rounded to FP32, compensated sums.  Each of the two roundings left (product,
    result) is uniform within 2^-24 of its value at most, sqrt(1/3) of that in the
    mean square; terms of zero mean, so |error| <= sqrt(2/3) 2^-24 |result| over
    all segments.  Plain sums of 20 and more terms are past that."""
    torch, lib, _ = env
    rng = np.random.default_rng(7)
    nseg = 40000
    # lanes' own segments up to 48 entries, the warp's from 49 on, several of each side by side, windows of 512
    lens = np.full(nseg, length) if length != "uneven" else rng.choice(
        [0, 1, 2, 5, 9, 16, 31, 33, 48, 49, 64, 130], nseg, p=[.1, .1, .1, .1, .2, .1, .1, .05, .05, .05, .04, .01])
    nnz = int(lens.sum())
    assert nnz < 32 * nseg
    idx = rng.integers(0, 9000, nnz)
    val, vec = rng.standard_normal(nnz).astype(np.float32), rng.standard_normal(9000).astype(np.float32)
    out = _spmv(torch, lib, lens, idx, val, vec)
    ref = np.bincount(np.repeat(np.arange(nseg), lens), weights=val.astype(np.float64) * vec[idx], minlength=nseg)
    assert np.linalg.norm(out - ref) <= np.sqrt(2 / 3) * 2.0**-24 * np.linalg.norm(ref)


def test_spmv_by_stream_keeps_infinities_and_nan(env):
    """Infinite and NaN entries of the vector, in segments of a lane and of a
    warp: the sums that plain additions give."""
    torch, lib, _ = env
    rng = np.random.default_rng(8)
    nseg = 40000
    lens = rng.choice([1, 2, 7, 30, 60, 700], nseg, p=[.3, .3, .2, .15, .045, .005])
    nnz = int(lens.sum())
    assert nnz < 32 * nseg
    vec = rng.standard_normal(5000).astype(np.float32)
    vec[:3] = np.inf, -np.inf, np.nan
    idx = rng.integers(3, 5000, nnz)
    odd = rng.choice(nnz, 9000, replace=False)
    idx[odd] = rng.integers(0, 3, 9000)
    val = rng.standard_normal(nnz).astype(np.float32)
    out = _spmv(torch, lib, lens, idx, val, vec)
    with np.errstate(invalid="ignore"):
        prod = val.astype(np.float64) * vec[idx]
        ref = np.bincount(np.repeat(np.arange(nseg), lens), weights=prod, minlength=nseg)
    assert np.isposinf(ref).any() and np.isneginf(ref).any() and np.isnan(ref).any()
    for f in (np.isposinf, np.isneginf, np.isnan):
        np.testing.assert_array_equal(f(out), f(ref))


@pytest.mark.parametrize("way", ["stream", "groups"])
def test_spmv_of_the_most_entries_an_int_counts(env, way):
    """2^31 - 1 entries: the last step of a lane group and the last window of the
    stream end past the largest int, and read nothing there."""
    torch, lib, _ = env
    nnz = 2**31 - 1
    if torch.cuda.mem_get_info()[0] < 24 * 2**30:
        pytest.skip("needs 18 GB on the device")
    nseg = nnz // 31 if way == "stream" else 20001
    ptr = torch.arange(nseg + 1, dtype=torch.int64, device="cuda") * (nnz // nseg)
    ptr[-1] = nnz  # the last segment takes the remainder
    idx = torch.zeros(nnz, dtype=torch.int32, device="cuda")
    val = torch.zeros(nnz, dtype=torch.float32, device="cuda")
    if way == "stream":
        val.fill_(1.0)  # sums: the lengths
        ref = torch.diff(ptr).float()
    else:  # the last 77 entries of every segment count
        for k in range(1, 78):
            val[ptr[1:] - k] = 1.0
        ref = torch.full((nseg,), 77.0, device="cuda")
    ptr = ptr.to(torch.int32)
    vec, out = torch.ones(4, device="cuda"), torch.full((nseg,), 7.0, device="cuda")
    assert lib.sih_pdhg_launch_csr_spmv(nseg, ptr.data_ptr(), idx.data_ptr(), val.data_ptr(), vec.data_ptr(),
                                        out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    del idx, val, ptr
    torch.cuda.empty_cache()
