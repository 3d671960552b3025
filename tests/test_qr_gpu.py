"""The fixed-effects design's factorisation on the GPU: the projection that a REML call leaves on the handle
against NumPy's FP64 basis, and what it refuses."""
import numpy as np
import pytest

from slemm_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu


def _problem(n, c, seed):
    counts, _ = synth.simulate_counts(n, 96, seed=seed)
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, c))
    X[:, 0] = 1.0
    if c > 2:
        X[:, 2] = X[:, 1] + 1e-3 * X[:, 2]
        X[:, 1:] *= 10.0 ** rng.uniform(-1, 1, c - 1)
    rvec = rng.uniform(0.3, 3.0, n).astype(np.float32)
    return synth.encode_bed(counts), X.astype(np.float32), rvec, rng.standard_normal(n).astype(np.float32)


# 16 blocks of 512 threads take 8,192 rows a sweep
@pytest.mark.parametrize("n,c", [(60, 1), (600, 2), (8191, 5), (8193, 33), (20001, 3)])
def test_projection_left_by_a_fit(gpu, n, c):
    rows, X, rvec, y = _problem(n, c, seed=n + c)
    rr = (np.float32(1) / np.sqrt(rvec)).astype(np.float32)
    Q = np.linalg.qr((rr[:, None] * X).astype(np.float64))[0]
    v = np.random.default_rng(1).standard_normal((n, 2)).astype(np.float32)
    with api.Genotypes(rows, n) as g:
        g.REML_grad(rvec, X, y, np.ones(96, np.float32), None, None, 0.4, 0.6, n_V=2)
        out = g.op(_lib.OP_QUADFORM, v, 0.0).astype(np.float64)
        g.set_projection(np.zeros((n, 1), np.float32))
        free = g.op(_lib.OP_QUADFORM, v - (Q @ (Q.T @ v)).astype(np.float32), 0.0).astype(np.float64)
    # FP32 entries of Q (2^-24 each), c of them, and the output's own rounding
    tol = (c + 8) * 2.0 ** -22 * np.linalg.norm(free, axis=0)
    assert np.all(np.abs(Q.T @ out) <= tol)
    assert np.all(np.linalg.norm(out - (free - Q @ (Q.T @ free)), axis=0) <= 2e-5 * np.linalg.norm(free, axis=0))


def test_designs_that_are_refused(gpu):
    n = 700
    rows, X, rvec, y = _problem(n, 4, seed=5)
    one = np.ones(96, np.float32)
    v = np.random.default_rng(1).standard_normal((n, 1)).astype(np.float32)
    twice, nan, inf, zero = X.copy(), X.copy(), X.copy(), X.copy()
    twice[:, 3] = 2 * X[:, 1]
    nan[n - 1, 2], inf[0, 0] = np.nan, np.inf
    zero[:, 1:] = 0.0
    with api.Genotypes(rows, n) as g:
        g.REML_grad(rvec, X, y, one, None, None, 0.4, 0.6, n_V=2)
        before = g.op(_lib.OP_QUADFORM, v, 0.5)
        for bad, code in ((twice, -5), (zero, -5), (nan, -6), (inf, -6)):
            for call in (lambda: g.REML_grad(rvec, bad, y, one, None, None, 0.4, 0.6, n_V=2),
                         lambda: g.LMC_REML(rvec, bad, y, one), lambda: g.SLDF_REML(rvec, bad, y, one, n_V=3)):
                with pytest.raises(_lib.SlemmError) as e:
                    call()
                assert e.value.code == code
        for bad in (twice, zero, nan, inf):
            with pytest.raises(_lib.SlemmError) as e:
                g.weighted_least_squares(rvec, bad, y)
            assert e.value.code == -1
        assert np.array_equal(before, g.op(_lib.OP_QUADFORM, v, 0.5))   # the handle is as it was


def test_refused_gradient_weights_leave_the_handle(gpu):
    """Window weights whose product with a SNP's own weight overflows are refused, and the handle keeps its
    weights and its projection."""
    n = 700
    rows, X, rvec, y = _problem(n, 3, seed=6)
    _, X2, rvec2, _ = _problem(n, 4, seed=7)
    v = np.random.default_rng(1).standard_normal((n, 2)).astype(np.float32)
    persnp = np.ones(96, np.float32)
    persnp[0] = 1000
    with api.Genotypes(rows, n) as g:
        g.REML_grad(rvec, X, y, np.ones(96, np.float32), None, None, 0.4, 0.6, n_V=2)
        before = [g.op(_lib.OP_QUADFORM, v, 0.5), g.op(_lib.OP_LDET, v, 0.5)]
        with pytest.raises(_lib.SlemmError):
            g.REML_grad(rvec2, X2, y, persnp, np.zeros(96, np.int32), np.full(1, 3e38, np.float32), 0.4, 0.6, n_V=2)
        for a, kind in zip(before, (_lib.OP_QUADFORM, _lib.OP_LDET)):
            assert np.array_equal(a, g.op(kind, v, 0.5))
