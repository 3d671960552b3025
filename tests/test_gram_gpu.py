"""The projected Gram blocks and their batched systems (--lmm windows, slemm_gwa blocks) against the
oracle, at the edges of the 128-column panels, of the 160- and 80-column operand groups and of the
256-row product tiles, with and without residual weights."""
import math

import numpy as np
import pytest

from oracle import slemm_np as orc
from slemm_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _data(n, m, c, weighted, seed):
    counts, _ = synth.simulate_counts(n, m, seed=seed)
    rng = np.random.default_rng(seed)
    rvec = rng.uniform(0.3, 3.0, n).astype(np.float32) if weighted else np.ones(n, np.float32)
    X = np.column_stack([np.ones(n)] + [rng.standard_normal(n) for _ in range(c - 1)]).astype(np.float32)
    return counts, synth.encode_bed(counts), rng.standard_normal(n).astype(np.float32), rvec, X


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("ws,n,c", [(2, 300, 1), (126, 700, 2), (128, 700, 0), (130, 1025, 3), (256, 700, 20),
                                    (322, 700, 2)])
def test_lmm_windows_at_panel_edges(gpu, weighted, ws, n, c):
    m = 600
    counts, rows, Py, rvec, X = _data(n, m, max(c, 1), weighted, seed=ws + n)
    gm = orc.genotype_mean(orc.popcounts(counts), n)
    gw = orc.snp_weights(gm, np.ones(m, np.float32))
    rr = (1 / np.sqrt(rvec)).astype(np.float32)
    Q = orc.qr_colpiv(rr[:, None] * X)[0][:, :c]
    ref = orc.LMM_quadforms(counts, Py, rr, Q, gm, gw, 1.7, num_qf=9, window_size=ws)
    with api.Genotypes(rows, n) as g:
        g.set_weights(gm, gw, rr)
        g.set_projection(Q.astype(np.float32))
        r = g.LMM_quadforms(Py, 1.7, num_qf=9, window_size=ws)
    assert r["variants"] == ref["variants"]
    # FP32 Gram entries (2^-22 of the diagonal) in systems whose condition number is a few: the ridge
    # is at least the diagonal's size here
    assert np.allclose(r["xBx"], ref["xBx"], rtol=2e-5, atol=0)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("block,n,c", [(4, 300, 1), (128, 1025, 2), (130, 700, 17), (322, 700, 2)])
def test_gwa_blocks_at_panel_edges(gpu, weighted, block, n, c):
    m, n_model = 1200, 500
    counts, rows, y, R, X = _data(n, m, c, weighted, seed=block + n)
    model = np.sort(np.random.default_rng(block).permutation(m)[:n_model])
    ref = orc.gwa_windows(2 - counts, y, R, X, model, 0, m - 1, block, 1.5, n_model, 0.9, 0.4, 20)
    with api.Genotypes(rows, n) as g:
        got = g.gwa_windows(y, R, X, model, 0, m - 1, block, 1.5, n_model, 0.9, 0.4, 20)
    ok = np.isfinite(ref[3])
    assert np.array_equal(ok, np.isfinite(got[3]))
    # the oracle is the script's float32: a few hundred FP32 products and sums per entry on both sides
    for a, b in zip(got[:3], ref[:3]):
        assert np.allclose(a[ok], b[ok], rtol=1e-3, atol=1e-5 * np.abs(b[ok]).max())


@pytest.mark.parametrize("ntest,mac", [(9, 0), (127, 60), (128, 60), (129, 200), (384, 60), (385, 10 ** 6)])
def test_gwa_statistics_of_the_tested_range(gpu, ntest, mac):
    """The last step of slemm_gwa: which variants are dropped, and β, se, χ² and p of the others from each
    other, for ranges at the edges of a block of 128 variants that do not start at SNP 0."""
    n, m, begin = 300, 400, 7
    counts, rows, y, _, X = _data(n, m, 2, False, seed=ntest)
    model = np.arange(begin, begin + ntest, max(1, ntest // 60))
    cfactor, snp_var = np.float32(0.9), np.float32(0.4)
    with api.Genotypes(rows, n) as g:
        beta, se, chisq, p = g.gwa_windows(y, None, X, model, begin, begin + ntest - 1, 40, 1.5, model.size, cfactor,
                                           snp_var, mac)
    s2 = counts[begin:begin + ntest].sum(1, dtype=np.int64)
    drop = np.minimum(s2, 2 * n - s2) <= mac
    for v in (beta, se, chisq, p):
        assert v.shape == (ntest,) and np.array_equal(np.isnan(v), drop)
    ok = ~drop
    z = beta[ok] / se[ok]   # IEEE FP32 on both sides
    assert np.array_equal(chisq[ok], z * z)
    # two complementary error functions (CUDA's and the C library's) of at most 5 units in the last place each
    want = np.array([math.erfc(math.sqrt(float(x) / 2)) for x in chisq[ok]])
    assert np.allclose(p[ok], want, rtol=10 * 2.0 ** -52, atol=0)


def _gwa_fp64(a2, y, R, X, model, block, tau, model_ct):
    """β (times 1/cfactor) and xx/τ of every variant in FP64; rr and the variants' means as FP32 values."""
    m, n = a2.shape
    rr = (np.float32(1) / np.sqrt(R)).astype(np.float64)
    Q = np.linalg.qr(rr[:, None] * X.astype(np.float64))[0]
    mean = (a2.sum(1, dtype=np.int64).astype(np.float32) / np.float32(n)).astype(np.float64)
    z = a2 - mean[:, None]
    Z = z * rr
    Z -= (Z @ Q) @ Q.T
    xx = np.empty(m)
    blocks, bounds, _ = orc.gwa_blocks(model, block, 0, m - 1)
    for blk, (lo, hi) in zip(blocks, bounds):
        B, mu = Z[blk], mean[blk]
        H = B @ B.T + np.diag(model_ct * tau * (2 - mu) * mu / 2)
        W = Z[lo:hi] @ B.T
        xx[lo:hi] = (Z[lo:hi] ** 2).sum(1) - np.einsum("ij,ij->i", W, np.linalg.solve(H, W.T).T)
    xx /= tau
    return -(z @ y.astype(np.float64)) / xx, xx


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("block,n,c", [(4, 300, 1), (128, 1025, 2), (130, 700, 17), (322, 700, 2)])
def test_gwa_blocks_vs_fp64(gpu, weighted, block, n, c):
    m, n_model = 1200, 500
    counts, rows, y, R, X = _data(n, m, c, weighted, seed=block + n)
    model = np.sort(np.random.default_rng(block).permutation(m)[:n_model])
    beta64, xx64 = _gwa_fp64(counts, y, R, X, model, block, 1.5, n_model)
    with api.Genotypes(rows, n) as g:
        beta, se, _, _ = g.gwa_windows(y, R, X, model, 0, m - 1, block, 1.5, n_model, 1.0, 1.0, -1)
    # FP32 Gram entries (2^-22 of the diagonal) in well-conditioned systems of up to 322 unknowns: xx to 1e-5
    assert np.allclose(1 / se.astype(np.float64) ** 2, xx64, rtol=1e-5, atol=0)
    assert np.allclose(beta, beta64, rtol=1e-5, atol=1e-5 * np.abs(beta64).max())


# weights over a factor of 100 of every size, and of two sizes; half of the variants in the individuals of small weight alone
@pytest.mark.parametrize("n", [2000, 20000])
@pytest.mark.parametrize("two", [False, True])
def test_gwa_rare_variants_of_small_weights(gpu, n, two):
    m, n_model = 600, 300
    rng = np.random.default_rng(3)
    counts = rng.binomial(2, rng.uniform(0.05, 0.5, m)[:, None], (m, n)).astype(np.uint8)
    R = (np.where(np.arange(n) % 2, 1.0, 100.0) if two else 10.0 ** rng.uniform(-2, 2, n)).astype(np.float32)
    counts[::2] *= R > np.median(R) if not two else R > 50
    y = rng.standard_normal(n).astype(np.float32)
    X = np.column_stack([np.ones(n), rng.standard_normal(n)]).astype(np.float32)
    model = np.sort(rng.permutation(m)[:n_model])
    _, xx64 = _gwa_fp64(counts, y, R, X, model, 100, 1.5, n_model)
    with api.Genotypes(synth.encode_bed(counts), n) as g:
        _, se, _, _ = g.gwa_windows(y, R, X, model, 0, m - 1, 100, 1.5, n_model, 1.0, 1.0, -1)
    # half of the variants are none of the model's, and their xx no small difference: FP32 entries and products, 2^-23 each,
    # give its relative error of a few of them
    assert np.median(np.abs(1 / se.astype(np.float64) ** 2 - xx64) / xx64) <= 4 * 2.0 ** -23


def test_lmm_windows_with_a_zero_weight(gpu):
    """A SNP of weight 0 has an infinite ridge: the markers whose windows hold it have no xBx, the others are as
    without it."""
    n, m, ws = 700, 600, 130
    counts, rows, Py, _, _ = _data(n, m, 1, False, seed=4)
    gm = orc.genotype_mean(orc.popcounts(counts), n)
    gw = orc.snp_weights(gm, np.ones(m, np.float32))
    got = []
    with api.Genotypes(rows, n) as g:
        g.set_projection(np.full((n, 1), 1 / np.sqrt(n), np.float32))
        for at in (None, 300):
            if at is not None:
                gw[at] = 0
            g.set_weights(gm, gw)
            got.append(g.LMM_quadforms(Py, 1.7, num_qf=20, window_size=ws))
    start = np.clip(np.array(got[0]["variants"]) - ws // 2, 0, m - ws)
    holds = (start <= 300) & (300 < start + ws)
    assert 0 < holds.sum() < holds.size
    a, b = got[0]["xBx"], got[1]["xBx"]
    assert np.array_equal(np.isnan(b), holds) and np.array_equal(a[~holds], b[~holds])


@pytest.mark.parametrize("weighted", [False, True])
def test_columns_of_wide_range(gpu, weighted):
    """Phenotypes and covariates over sixteen orders of magnitude: more digits than short calls queue at first."""
    n, m, n_model, block = 700, 300, 120, 40
    counts, rows, y, R, X = _data(n, m, 2, weighted, seed=11)
    rng = np.random.default_rng(2)
    y = (y * 10.0 ** rng.uniform(-8, 8, n)).astype(np.float32)
    X[:, 1] *= (10.0 ** rng.uniform(-16, 0, n)).astype(np.float32)   # beside an intercept: of full rank
    model = np.sort(rng.permutation(m)[:n_model])
    beta64, xx64 = _gwa_fp64(counts, y, R, X, model, block, 1.5, n_model)
    gm = orc.genotype_mean(orc.popcounts(counts), n)
    gw = orc.snp_weights(gm, np.ones(m, np.float32))
    rr = (1 / np.sqrt(R)).astype(np.float32)
    Q = np.linalg.qr(rr[:, None] * X.astype(np.float64))[0]
    ref = orc.LMM_quadforms(counts, y, rr, Q, gm, gw, 1.7, num_qf=9, window_size=130)
    with api.Genotypes(rows, n) as g:
        beta, se, _, _ = g.gwa_windows(y, R, X, model, 0, m - 1, block, 1.5, n_model, 1.0, 1.0, -1)
        g.set_weights(gm, gw, rr)
        g.set_projection(Q.astype(np.float32))
        r = g.LMM_quadforms(y, 1.7, num_qf=9, window_size=130)
    # the bounds of the tests above
    assert np.allclose(1 / se.astype(np.float64) ** 2, xx64, rtol=1e-5, atol=0)
    assert np.allclose(beta, beta64, rtol=1e-5, atol=1e-5 * np.abs(beta64).max())
    assert np.allclose(r["xBx"], ref["xBx"], rtol=2e-5, atol=0)
