"""GEBV and the GWAS score terms against extended- and double-precision sums, at the edges of the
exact product's tiles and of its 8,192-element partial sums."""
import numpy as np
import pytest

from conftest import make_case
from slemm_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (257, 127), (300, 8192), (129, 8193), (1000, 16640)])
def test_gebv_exact_products(gpu, n, m):
    from slemm_gb300 import api
    rows, _, dec = make_case(n, m, seed=n + m, missing=0.02)
    rng = np.random.default_rng(m)
    alpha = rng.standard_normal(m) * 10.0 ** rng.uniform(-12, 2, m)
    flip = (rng.random(m) < 0.5).astype(np.uint8)
    with api.Genotypes(rows, n) as g:
        got = g.gebv(alpha, flip)
    x = dec.astype(np.longdouble)
    want = (np.where(flip[:, None] == 1, 2 - x, x) * alpha.astype(np.longdouble)[:, None]).sum(0)
    # the slices resolve 2^-65 of max|alpha|; the shift 2·Σalpha is a running FP64 sum of m terms and
    # the last combination rounds a few times
    assert np.abs(got - want).max() <= 2.0 ** -52 * 4 * m * np.abs(alpha).max()


@pytest.mark.parametrize("value", [0.7, -1.0, 2.0 ** -1060, 1e300])
def test_gebv_largest_partial_sums(gpu, value):
    """Every count 2 and every effect the same: the partial sums reach their bound of 2^24."""
    from slemm_gb300 import api
    n, m = 130, 8192 + 64
    with api.Genotypes(synth.encode_bed(np.full((m, n), 2, np.uint8)), n) as g:
        got = g.gebv(np.full(m, value))
    want = 2.0 * m * value
    assert np.abs(got - want).max() <= 2.0 ** -51 * abs(want)


@pytest.mark.parametrize("n,m,c,unit", [(255, 1, 0, False), (8192, 130, 1, False), (8200, 257, 14, False),
                                        (20001, 300, 3, False), (8200, 257, 14, True), (513, 129, 0, True)])
def test_score_terms_exact_products(gpu, n, m, c, unit):
    from slemm_gb300 import api
    rows, _, dec = make_case(n, m, seed=n + c, missing=0.01)
    rng = np.random.default_rng(n)
    y = (rng.standard_normal(n) * 3 + 1).astype(np.float32)
    rr = np.ones(n, np.float32) if unit else (1 / np.sqrt(10.0 ** rng.uniform(-3, 3, n))).astype(np.float32)
    X = np.column_stack([np.ones(n)] + [rng.standard_normal(n) for _ in range(c)])[:, :c]
    Q = np.linalg.qr(rr[:, None] * X)[0].astype(np.float32) if c else np.zeros((n, 0), np.float32)
    x = dec.astype(np.float64)
    gm = x.mean(1)
    with api.Genotypes(rows, n) as g:
        g.set_weights(gm.astype(np.float32), np.ones(m, np.float32), rr)
        g.set_projection(Q)
        xy, xx = g.score_terms(y, 0)
        bad = y.copy()
        bad[n // 2] = np.nan
        nan_xy, same_xx = g.score_terms(bad, 0)
    z = x - gm[:, None]
    want_xy = -(z @ y.astype(np.float64))
    # the columns as the kernel takes them: rr·Q_l and rr² rounded to FP32
    r2 = (rr * rr).astype(np.float64)
    rq = (rr[:, None] * Q).astype(np.float64)
    want_xx = (z * z) @ r2 - ((z @ rq) ** 2).sum(1)
    # FP32 rounding of the result, and the FP64 cancellation of the centring terms
    assert np.all(np.abs(xy - want_xy) <= 2.0 ** -23 * np.abs(want_xy) + 1e-12 * np.abs(y).sum())
    assert np.all(np.abs(xx - want_xx) <= 2.0 ** -23 * np.abs(want_xx) + 1e-12 * r2.sum())
    assert np.all(np.isnan(nan_xy)) and np.array_equal(same_xx, xx)


@pytest.mark.parametrize("small", [1e-6, 1e-14, 1e-40, 1e-300])
def test_gebv_small_effects_beside_a_large_one(gpu, small):
    """Individuals without a copy of the SNP of the large effect: their sum of small effects is as accurate as
    without it."""
    from slemm_gb300 import api
    n, m = 700, 300
    rows, _, dec = make_case(n, m, seed=9)
    rng = np.random.default_rng(5)
    alpha = rng.uniform(0.5, 1.0, m) * small
    alpha[7] = 1.0
    alpha[11] = 0.0
    assert (dec[7] == 0).sum() > 10
    with api.Genotypes(rows, n) as g:
        got = g.gebv(alpha)
    want = (dec.astype(np.longdouble) * alpha.astype(np.longdouble)[:, None]).sum(0)
    # exact sums of positive terms, rounded a few times at the end
    assert np.all(np.abs(got - want) <= 2.0 ** -51 * want)


@pytest.mark.parametrize("n,m,c", [(700, 300, 2), (8200, 257, 14)])
def test_score_terms_with_far_smaller_weights(gpu, n, m, c):
    """Rare variants carried by individuals of small weight alone: what is left of xx after the centring terms
    of the large weights has FP64's accuracy."""
    from slemm_gb300 import api
    rng = np.random.default_rng(n)
    rr = np.where(np.arange(n) < 40, 1.0, rng.uniform(0.5, 1.0, n) * 1e-12).astype(np.float32)
    dec = rng.binomial(2, 0.3, (m, n)).astype(np.uint8)
    dec[:, :40] = 0
    y = (rng.standard_normal(n) * 10.0 ** rng.uniform(-12, 12, n)).astype(np.float32)
    y[:40] = 0
    Q = np.zeros((n, c), np.float32)
    Q[np.arange(c), np.arange(c)] = 1                     # the projection takes the first c individuals out
    x = dec.astype(np.float64)
    gm = x.mean(1)
    with api.Genotypes(synth.encode_bed(dec), n) as g:
        g.set_weights(gm.astype(np.float32), np.ones(m, np.float32), rr)
        g.set_projection(Q)
        xy, xx = g.score_terms(y, 0)
    z = (x - gm[:, None]).astype(np.longdouble)
    want_xy = -(z @ y.astype(np.longdouble))
    r2 = (rr * rr).astype(np.longdouble)
    rq = (rr[:, None] * Q).astype(np.longdouble)
    want_xx = (z * z) @ r2 - ((z @ rq) ** 2).sum(1)
    # FP64 sums of the terms, then FP32
    size = (z * z) @ r2 + ((np.abs(z) @ np.abs(rq)) ** 2).sum(1)
    assert np.all(np.abs(xy - want_xy) <= 2.0 ** -23 * np.abs(want_xy) + 2.0 ** -50 * (np.abs(z) @ np.abs(y).astype(np.longdouble)))
    assert np.all(np.abs(xx - want_xx) <= 2.0 ** -23 * np.abs(want_xx) + 2.0 ** -50 * size)


def test_score_terms_of_rare_variants_with_small_weights(gpu):
    """Variants carried by individuals of small weight alone, in a sample whose weight is one individual's: the
    carriers' part of xx, 2^-46 of the largest weight each, is comparable with the centring terms."""
    from slemm_gb300 import api
    n, m = 100003, 40
    rng = np.random.default_rng(3)
    rr = (rng.uniform(0.5, 1.0, n) * 2.0 ** -23).astype(np.float32)
    rr[77] = 1
    dec = np.zeros((m, n), np.uint8)
    for j in range(m):
        dec[j, rng.choice(np.arange(100, n), 25, replace=False)] = 1
    y = rng.standard_normal(n).astype(np.float32)
    with api.Genotypes(synth.encode_bed(dec), n) as g:
        g.set_weights(dec.mean(1).astype(np.float32), np.ones(m, np.float32), rr)
        g.set_projection(np.zeros((n, 0), np.float32))
        _, xx = g.score_terms(y, 0)
    z = (dec - dec.mean(1, dtype=np.float64)[:, None]).astype(np.longdouble)
    want = (z * z) @ (rr * rr).astype(np.longdouble)
    # FP64 sums of positive terms, then FP32
    assert np.all(np.abs(xx - want) <= 2.0 ** -23 * want)


@pytest.mark.parametrize("bits", [30, 36, 37, 60, 200])
@pytest.mark.parametrize("unit", [False, True])
def test_score_terms_of_every_range(gpu, bits, unit):
    """Short calls guess the columns' digits: phenotypes whose values span up to 2^200, below and above what the guess
    holds, have the sums of the plain product."""
    from slemm_gb300 import api
    n, m = 515, 130
    rows, _, dec = make_case(n, m, seed=bits)
    rng = np.random.default_rng(bits)
    y = np.zeros(n, np.float32)
    y[:256] = 1.5 * 2.0 ** -(bits - 24)          # a tiny value and its carriers beside one large value
    y[300] = 2.0 ** 24
    y[301] = -2.0 ** 24                          # of two individuals with the same genotypes
    dec = dec.copy()
    dec[:, 301] = dec[:, 300]
    rr = np.ones(n, np.float32) if unit else rng.uniform(0.5, 2.0, n).astype(np.float32)
    with api.Genotypes(synth.encode_bed(dec), n) as g:
        g.set_weights(dec.mean(1).astype(np.float32), np.ones(m, np.float32), rr)
        g.set_projection(np.zeros((n, 0), np.float32))
        xy, _ = g.score_terms(y, 0)
    z = dec.astype(np.float64) - dec.mean(1, dtype=np.float64)[:, None]
    want = -(z[:, :256].sum(1) * np.float64(y[0]))
    # the large pair cancels in the exact sums; the total that centres them is an FP64 sum
    assert np.all(np.abs(xy - want) <= 2.0 ** -23 * np.abs(want) + 2.0 ** -50 * (np.abs(z) @ np.abs(y).astype(np.float64)))
