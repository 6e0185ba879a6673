"""Batched GPU ICP against the oracle's restatement of the reference's PCL
point-to-point ICP (parity is unpinned against PCL itself, which is not
available): transforms agree within a stated rotation / translation
tolerance and the registration MSE agrees to 2 % (FP32 nearest neighbours
and Kahan-compensated FP32 sums on the GPU, FP64 throughout in the oracle)."""
import numpy as np
import pytest

ROT_TOL_DEG = 0.1      # GPU vs oracle final rotation
TRANS_TOL_VOX = 0.1    # GPU vs oracle final translation, at the source centroid
MSE_RTOL = 0.02        # GPU vs oracle fitness score


def _pairs(pvvc_lib, n, seed):
    from pvvc.icp import make_pairs
    return make_pairs(n, seed=seed)


def _trans_err(A, B, pairs):
    c = np.array([s.mean(0) for s in pairs.src])
    pa = np.einsum("nij,nj->ni", A[:, :3, :3], c) + A[:, :3, 3]
    pb = np.einsum("nij,nj->ni", B[:, :3, :3], c) + B[:, :3, 3]
    return np.linalg.norm(pa - pb, axis=1)


def test_oracle_icp_recovers_ground_truth(pvvc_lib, oracle):
    from pvvc.icp import rotation_error_deg
    pairs = _pairs(pvvc_lib, 6, 1)
    Ts, fits = [], []
    for s, t in zip(pairs.src, pairs.tgt):
        T, fit, it, conv = oracle.icp_align(s, t, max_iter=50, fitness_eps=0.0, transform_eps=0.0, mse_abs_eps=1e-6)
        assert conv  # the iteration cap counts as converged, as in PCL
        Ts.append(T)
        fits.append(fit)
    err = rotation_error_deg(np.array(Ts), pairs.T_true)
    # plain ICP from identity can stop in a local minimum; most pairs register
    assert np.median(err) < 0.5 and (np.array(fits) < 2.0).sum() >= 4


def test_oracle_cloud_mse_identity_is_zero(oracle):
    rng = np.random.default_rng(0)
    a = rng.integers(0, 100, (500, 3)).astype(np.float32)
    assert oracle.cloud_mse(a, a) == 0.0
    b = a + np.float32(1.0)
    assert abs(oracle.cloud_mse(a, b) - 3.0) < 1e-5 or oracle.cloud_mse(a, b) <= 3.0


CLOUD_MSE_RTOL = 1e-5  # the reference sums float distances in point order; the oracle (double) and GPU (compensated) do not


def _cloud_mse_golden():
    import os
    z = np.load(os.path.join(os.path.dirname(__file__), "golden", "cloud_mse.npz"))
    ao, bo = z["a_off"], z["b_off"]
    return [(z["a"][ao[i]:ao[i + 1]], z["b"][bo[i]:bo[i + 1]], float(z["mse"][i])) for i in range(len(z["mse"]))]


def test_oracle_cloud_mse_matches_reference(oracle):
    """Pinned against the reference's own ICPBase::CloudMSE (golden fixture
    from tests/golden/make_golden.py)."""
    for a, b, want in _cloud_mse_golden():
        got = oracle.cloud_mse(a, b)
        assert abs(got - want) <= CLOUD_MSE_RTOL * want, (got, want)


@pytest.mark.gpu
def test_gpu_cloud_mse_matches_reference(pvvc_lib):
    import torch
    from pvvc.icp import IcpBatch, Pairs
    cases = _cloud_mse_golden()
    b = IcpBatch(Pairs([c[0] for c in cases], [c[1] for c in cases], np.repeat(np.eye(4)[None], len(cases), 0)))
    T = torch.from_numpy(np.tile(np.eye(4, dtype=np.float32).reshape(16), (len(cases), 1))).cuda()
    got = b.cloud_mse(T)
    for i, (_, _, want) in enumerate(cases):
        assert abs(got[i] - want) <= CLOUD_MSE_RTOL * want, (i, got[i], want)


@pytest.mark.gpu
def test_gpu_icp_matches_oracle(pvvc_lib, oracle):
    import torch
    assert torch.cuda.is_available()
    from pvvc.icp import IcpBatch, rotation_error_deg
    pairs = _pairs(pvvc_lib, 48, 3)
    b = IcpBatch(pairs)
    b.run(max_iter=50, fitness_eps=0.0, transform_eps=0.0, mse_abs_eps=1e-6)
    T, mse, iters, conv = b.results()
    To, mo = [], []
    for s, t in zip(pairs.src, pairs.tgt):
        Tt, fit, it, cv = oracle.icp_align(s, t, max_iter=50, fitness_eps=0.0, transform_eps=0.0, mse_abs_eps=1e-6)
        To.append(Tt)
        mo.append(fit)
    To, mo = np.array(To), np.array(mo)
    assert conv.all()
    rot = rotation_error_deg(T, To)
    tr = _trans_err(T, To, pairs)
    assert (rot < ROT_TOL_DEG).mean() >= 0.95, rot
    assert (tr < TRANS_TOL_VOX).mean() >= 0.95, tr
    assert (np.abs(mse - mo) <= MSE_RTOL * mo + 1e-3).mean() >= 0.95, (mse, mo)


@pytest.mark.gpu
def test_gpu_cloud_mse_matches_oracle(pvvc_lib, oracle):
    import torch
    from pvvc.icp import IcpBatch
    pairs = _pairs(pvvc_lib, 16, 4)
    b = IcpBatch(pairs)
    T = torch.from_numpy(np.ascontiguousarray(pairs.T_true.reshape(-1, 16), np.float32)).cuda()
    got = b.cloud_mse(T)
    for i, (s, t) in enumerate(zip(pairs.src, pairs.tgt)):
        M = pairs.T_true[i].astype(np.float32)
        st = (s @ M[:3, :3].T + M[:3, 3]).astype(np.float32)
        want = oracle.cloud_mse(st, t)
        assert abs(got[i] - want) <= 1e-3 * want + 1e-4, (i, got[i], want)


@pytest.mark.gpu
def test_gpu_icp_edge_cases(pvvc_lib):
    """Tiny and degenerate pairs finish with a status instead of hanging."""
    import torch
    from pvvc.icp import IcpBatch, Pairs
    rng = np.random.default_rng(5)
    one = np.array([[1.0, 2.0, 3.0]], np.float32)
    two = np.array([[0, 0, 0], [5, 0, 0]], np.float32)
    line = np.stack([np.arange(50), np.zeros(50), np.zeros(50)], 1).astype(np.float32)
    cloud = rng.integers(0, 40, (300, 3)).astype(np.float32)
    pairs = Pairs([one, two, line, cloud], [one + 1, two, line + 2, cloud + 0.5], np.repeat(np.eye(4)[None], 4, 0))
    b = IcpBatch(pairs)
    b.run(max_iter=30)
    T, mse, iters, conv = b.results()
    assert not conv[0] and not conv[1]          # fewer than 3 correspondences
    assert np.isfinite(T).all() and (iters <= 30).all()
    assert conv[3] and mse[3] < 1.0


@pytest.mark.gpu
def test_gpu_icp_same_for_any_cta_size(pvvc_lib):
    """One batch of pairs, and the same pairs repeated until the launch takes
    smaller CTAs: a pair's results do not depend on the batch, bit for bit; and
    neither on the scratch for its neighbours (the entry point without one)."""
    import ctypes as C
    import torch
    from pvvc import _lib as L
    from pvvc.icp import IcpBatch, Pairs
    base = _pairs(pvvc_lib, 12, 7)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ref = None
    for reps in (1, 4 * sms // 12 + 1, 10 * sms // 12 + 1):
        p = Pairs(base.src * reps, base.tgt * reps, np.tile(base.T_true, (reps, 1, 1)))
        b = IcpBatch(p)
        b.run(max_iter=20)
        T, mse, iters, conv = b.results()
        got = (T.reshape(reps, 12, 16), mse.reshape(reps, 12), iters.reshape(reps, 12), conv.reshape(reps, 12))
        ref = ref or [g[0] for g in got]
        for g, w in zip(got, ref):
            assert (g == w[None]).all()
    b = IcpBatch(base)
    prm = L.IcpParams(1e6, 20, 0.0, 0.0, 1e-6)
    L.check(L.lib().pvvc_icp_batch_noalloc(b.n, b.src.data_ptr(), b.soff.data_ptr(), b.tgt.data_ptr(), b.toff.data_ptr(), None,
                                           C.byref(prm), b.T.data_ptr(), b.mse.data_ptr(), b.iters.data_ptr(),
                                           b.conv.data_ptr(), b.nt, torch.cuda.current_stream().cuda_stream), "noalloc")
    for g, w in zip(b.results(), ref):
        assert (g.reshape(w.shape) == w).all()


@pytest.mark.gpu
@pytest.mark.parametrize("noalloc", [False, True])
def test_gpu_icp_size_classes(pvvc_lib, noalloc):
    """More pairs than SMs, sources of 0 to 6,000 points around the limits of the
    size classes, in a shuffled order: every pair is run once, and its results
    are those of a batch that fits on the device, bit for bit."""
    import ctypes as C
    import torch
    from pvvc import _lib as L
    from pvvc.icp import IcpBatch, Pairs
    rng = np.random.default_rng(4)
    sizes = [0, 1, 3, 724, 725, 1024, 1025, 1448, 1449, 2047, 2048, 2896, 2897, 4095, 4096, 5792, 5793, 6000]
    sizes += [int(v) for v in rng.integers(3, 700, 40)]
    n, few = torch.cuda.get_device_properties(0).multi_processor_count + 40, 58
    order = rng.permutation(np.arange(n) % few)
    src = [rng.uniform(0, 40, (v, 3)).astype(np.float32) for v in sizes]
    tgt = [(s + rng.normal(0, 0.4, s.shape)).astype(np.float32)[: max(len(s), 1)] if len(s) else np.ones((3, 3), np.float32)
           for s in src]

    def results(ids):
        b = IcpBatch(Pairs([src[i] for i in ids], [tgt[i] for i in ids], np.tile(np.eye(4), (len(ids), 1, 1))))
        prm = L.IcpParams(1e6, 10, 0.0, 0.0, 1e-6)
        if noalloc:
            L.check(L.lib().pvvc_icp_batch_noalloc(b.n, b.src.data_ptr(), b.soff.data_ptr(), b.tgt.data_ptr(), b.toff.data_ptr(),
                                                   None, C.byref(prm), b.T.data_ptr(), b.mse.data_ptr(), b.iters.data_ptr(),
                                                   b.conv.data_ptr(), b.nt, torch.cuda.current_stream().cuda_stream), "noalloc")
        else:
            b.run(max_iter=10)
        return [np.asarray(v).reshape(len(ids), -1) for v in b.results()]

    want = results(range(few))
    for g, w in zip(results(order), want):
        assert np.array_equal(g, w[order], equal_nan=g.dtype.kind == "f")


@pytest.mark.gpu
@pytest.mark.parametrize("flat", [1.0, 1e-3, 0.0])
def test_gpu_icp_flat_patches(pvvc_lib, oracle, flat):
    """A patch and its moved copy, flattened to a plane: the covariance's
    smallest singular value goes to zero (the SVD takes over from the polar
    iteration)."""
    from pvvc.icp import IcpBatch, Pairs, rotation, rotation_error_deg
    rng = np.random.default_rng(11)
    s = np.unique(rng.integers(0, 60, (900, 3)), axis=0).astype(np.float64) * [1, 1, flat]
    R = rotation([0, 0, 1], 1.0)
    t = s @ R.T + [0.3, -0.2, 0.1 * flat]
    p = Pairs([s.astype(np.float32)], [t.astype(np.float32)], np.eye(4)[None])
    b = IcpBatch(p)
    b.run(max_iter=30)
    T, mse, _, _ = b.results()
    To, fit, _, _ = oracle.icp_align(p.src[0], p.tgt[0], max_iter=30, fitness_eps=0.0, transform_eps=0.0, mse_abs_eps=1e-6)
    assert rotation_error_deg(T, np.array([To]))[0] < ROT_TOL_DEG
    assert _trans_err(T, np.array([To]), p)[0] < TRANS_TOL_VOX
    assert abs(mse[0] - fit) <= MSE_RTOL * fit + 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("far", [30.0, 1e3, 1e6])
def test_gpu_icp_far_outliers(pvvc_lib, far):
    """Clouds with a point far off, which leaves the others in one or a few cells of
    the grid, between pairs without one: ICP with and without kept neighbours gives
    the same bits, each pair those it has alone, and the clouds' MSE is brute
    force's."""
    import ctypes as C
    import torch
    from pvvc import _lib as L
    from pvvc.icp import IcpBatch, Pairs
    rng = np.random.default_rng(6)
    src, tgt = [], []
    for i, n in enumerate((40, 66, 300, 700, 1500, 900)):
        s = rng.integers(0, 30, (n, 3)).astype(np.float32)
        t = (s + rng.normal(0, 0.4, s.shape)).astype(np.float32)
        if i != 3:
            t[-1] += np.float32(far)
            s[0] += np.float32(far if i % 2 else 0)
        src.append(s)
        tgt.append(t)

    def noalloc(b, iters):
        prm = L.IcpParams(1e6, iters, 0.0, 0.0, 1e-6)
        L.check(L.lib().pvvc_icp_batch_noalloc(b.n, b.src.data_ptr(), b.soff.data_ptr(), b.tgt.data_ptr(), b.toff.data_ptr(),
                                               None, C.byref(prm), b.T.data_ptr(), b.mse.data_ptr(), b.iters.data_ptr(),
                                               b.conv.data_ptr(), b.nt, torch.cuda.current_stream().cuda_stream), "noalloc")

    def batch(ids):
        return IcpBatch(Pairs([src[i] for i in ids], [tgt[i] for i in ids], np.tile(np.eye(4), (len(ids), 1, 1))))

    b = batch(range(6))
    b.run(max_iter=8)
    want = b.results()
    mse = b.cloud_mse()
    for v in (b.T, b.mse, b.iters, b.conv):
        v.zero_()
    noalloc(b, 8)
    for g, w in zip(b.results(), want):
        assert np.array_equal(g, w)
    for i in range(6):
        one = batch([i])
        noalloc(one, 8)
        for g, w in zip(one.results(), want):
            assert np.array_equal(g[0], w[i])
        m = (src[i].astype(np.float64) @ want[0][i, :3, :3].astype(np.float64).T + want[0][i, :3, 3]).astype(np.float32)
        d = ((m[:, None].astype(np.float64) - tgt[i][None]) ** 2).sum(2)
        # float32 coordinates of the size of `far`
        tol = 1e-5 * max(d.min(1).mean(), d.min(0).mean()) + 1e-5 + (4e-7 * far) ** 2 + 1e-6 * far
        assert abs(mse[i] - max(d.min(1).mean(), d.min(0).mean())) <= tol, i
