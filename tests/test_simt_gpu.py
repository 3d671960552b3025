"""The FP32 CUDA-core product: every kernel width, ragged sizes and the range of its staged scaling,
against FP64 sums."""
import numpy as np
import pytest

from conftest import make_case
from oracle import slemm_np as orc
from slemm_gb300 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(37, 5), (515, 130), (4100, 257)])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 8, 15])
@pytest.mark.parametrize("size", [1e-30, 1.0, 1e33])
def test_fp32_products_vs_fp64(gpu, n, m, k, size):
    rows, _, dec = make_case(n, m, seed=n + k)
    rng = np.random.default_rng(k)
    gm = orc.genotype_mean(orc.popcounts(dec), n)
    x = dec.astype(np.float64) - gm[:, None].astype(np.float64)
    v = (rng.standard_normal((n, k)) * size).astype(np.float32)
    u = (rng.standard_normal((m, k)) * size).astype(np.float32)
    v[:: max(1, n // 7)] *= np.float32(1e-6)          # small beside large in one stage
    u[0] = 0
    with api.Genotypes(rows, n) as g:
        g.set_weights(gm, np.ones(m, np.float32))
        g.set_precision(_lib.PREC_FP32)
        got = [g.rmatvec(v), g.matvec(u)]
    for a, b in zip(got, [x @ v.astype(np.float64), x.T @ u.astype(np.float64)]):
        # FP32 sums of 64 products, 2^-23 of the terms' size √(rows), and the centring's rounding
        assert np.linalg.norm(a - b) <= 2e-6 * np.linalg.norm(b)


@pytest.mark.parametrize("n,m", [(515, 130), (4100, 257)])
@pytest.mark.parametrize("k", [2, 3, 4, 8, 15])
def test_fp32_columns_of_different_sizes(gpu, n, m, k):
    """Columns from 1e-20 to 1e20 in one call, and columns that hold ∞ or NaN beside large finite ones: every
    column has the accuracy that it has alone."""
    rows, _, dec = make_case(n, m, seed=n + k)
    rng = np.random.default_rng(n + k)
    gm = orc.genotype_mean(orc.popcounts(dec), n)
    x = dec.astype(np.float64) - gm[:, None].astype(np.float64)
    size = 10.0 ** rng.permutation(np.linspace(-20, 20, k))
    v = (rng.standard_normal((n, k)) * size).astype(np.float32)
    u = (rng.standard_normal((m, k)) * size).astype(np.float32)
    with api.Genotypes(rows, n) as g:
        g.set_weights(gm, np.ones(m, np.float32))
        g.set_precision(_lib.PREC_FP32)
        got = [g.rmatvec(v), g.matvec(u)]
        for a, b in zip(got, [x @ v.astype(np.float64), x.T @ u.astype(np.float64)]):
            # the bound of test_fp32_products_vs_fp64, for each column
            assert np.all(np.linalg.norm(a - b, axis=0) <= 2e-6 * np.linalg.norm(b, axis=0))
        for bad in (np.inf, np.nan):
            w, t = v.copy(), u.copy()
            w[:, 1:] = 1e20 * rng.standard_normal((n, k - 1))
            t[:, 1:] = 1e20 * rng.standard_normal((m, k - 1))
            w[n // 2, 0] = t[m // 2, 0] = bad
            for a, b in zip([g.rmatvec(w), g.matvec(t)], [x @ w[:, 1:].astype(np.float64), x.T @ t[:, 1:].astype(np.float64)]):
                assert not np.isfinite(a[:, 0]).any()
                assert np.all(np.linalg.norm(a[:, 1:] - b, axis=0) <= 2e-6 * np.linalg.norm(b, axis=0))


@pytest.mark.parametrize("small", [1e-15, 1e-24, 1e-30, 1e-37])
@pytest.mark.parametrize("large", [1.0, 1e9, 1e30])
def test_fp32_small_terms_beside_a_large_one(gpu, small, large):
    """Individuals without a copy of the SNP of the large effect: their sums of small effects (no centring) are
    as accurate as without it."""
    n, m = 700, 300
    rows, _, dec = make_case(n, m, seed=9)
    rng = np.random.default_rng(5)
    u = (rng.uniform(0.5, 1.0, (m, 2)) * small).astype(np.float32)
    u[7, 0] = large
    with api.Genotypes(rows, n) as g:
        g.set_weights(np.zeros(m, np.float32), np.ones(m, np.float32))
        g.set_precision(_lib.PREC_FP32)
        got = g.matvec(u)
    want = dec.T.astype(np.float64) @ u.astype(np.float64)
    assert (dec[7] == 0).sum() > 10
    # positive terms: FP32 sums of 64, 2^-23 each
    assert np.all(np.abs(got - want) <= 64 * 2.0 ** -23 * want)
