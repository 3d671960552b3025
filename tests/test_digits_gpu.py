"""FP16X2 passes of at most 32 columns run on E4M3 digits: the operators against the FP64 oracle at the
edges of the digit plans (N = 48 … 160, the FP16 plan from 33 columns on), of the 16-row words and of
the 4-wide loads; the exact sums at their bound; and the bounded waits."""
import numpy as np
import pytest

from conftest import make_case
from oracle import slemm_np as orc
from slemm_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(4096 + 4, 1001), (3001, 516), (17, 300), (8192, 4099)])
@pytest.mark.parametrize("k", [1, 8, 9, 12, 13, 24, 32, 33])
def test_digit_operators_vs_oracle(gpu, n, m, k):
    rows, _, dec = make_case(n, m, seed=n + k)
    rng = np.random.default_rng(k)
    gm = orc.genotype_mean(orc.popcounts(dec), n)
    w = orc.snp_weights(np.clip(gm, 0.02, 1.98), np.ones(m, np.float32))
    rr = rng.uniform(0.5, 2.0, n).astype(np.float32)
    Q = np.linalg.qr(rr[:, None] * np.column_stack([np.ones(n), rng.standard_normal(n)]))[0].astype(np.float32)
    ref = orc.Operators(dec, gm, w, rr, Q, dtype=np.float64)
    v = (rng.standard_normal((n, k)) * 10.0 ** rng.uniform(-20, 20, k)).astype(np.float32)
    v[:, 0] += 100 * np.abs(v[:, 0]).max()          # a column with a large mean
    if k > 1:
        v[:, 1] = 0                                 # an empty column
    u = rng.standard_normal((m, k)).astype(np.float32)
    with api.Genotypes(rows, n) as g:
        g.set_weights(gm, w, rr)
        g.set_projection(Q)
        got = [g.H0_quadform_mv(0.4, v), g.H0_ldet_mv(0.4, v), g.rmatvec(v), g.weighted_rmatvec(v), g.matvec(u)]
    want = [ref.H0_quadform_mv(0.4, v), ref.H0_ldet_mv(0.4, v), ref.rmatvec(v), ref.weighted_rmatvec(v), ref.matvec(u)]
    for a, b in zip(got, want):
        err = np.linalg.norm(a - b, axis=0)
        scale = np.linalg.norm(b, axis=0)
        # the operators' tolerance of the FP16X2 precision; the centred constant part of column 0 is a
        # difference of sums 100 times its size
        assert np.all(err <= 2e-6 * scale + (np.arange(k) == 0) * 2e-4 * scale)


def test_exact_sums_at_their_bound(gpu):
    """2^19 counts of 2 against the largest digit: every partial sum reaches 2^24."""
    n, m = 130, (1 << 19) + 64
    rows = np.full((m, (n + 3) // 4), 0xFF, np.uint8)
    with api.Genotypes(rows, n) as g:
        assert np.array_equal(g.gebv(np.full(m, 15.99)), np.full(n, g.gebv(np.full(m, 15.99))[0]))
        got = g.gebv(np.full(m, -15.75))            # digits −16 and 8: the leading one at its bound
    assert np.array_equal(got, np.full(n, -15.75 * 2 * m))


@pytest.mark.parametrize("k", [1, 24])
def test_withheld_digit_copy_times_out_and_handle_recovers(gpu, k):
    n, m = 3001, 1537
    rows, _, dec = make_case(n, m, seed=62)
    gm = orc.genotype_mean(orc.popcounts(dec), n)
    w = orc.snp_weights(gm, np.ones(m, np.float32))
    v = np.random.default_rng(k).standard_normal((n, k)).astype(np.float32)
    want = orc.Operators(dec, gm, w, None, None, dtype=np.float64).rmatvec(v)
    with api.Genotypes(rows, n) as g:
        g.set_weights(gm, w)
        _lib.check(gpu.slemm_gpu_test_withhold_b_stage(0))
        with pytest.raises(_lib.SlemmError) as e:
            g.rmatvec(v)
        assert e.value.code == -2 and "bounded wait" in str(e.value)
        got = g.rmatvec(v)
        assert np.linalg.norm(got - want) / np.linalg.norm(want) < 2e-6


@pytest.mark.parametrize("which", ["rmatvec", "matvec"])
@pytest.mark.parametrize("size", [8.6e37, 1.05e38, 1.7e38])
def test_columns_near_the_largest_float(gpu, size, which):
    """One large entry, whose products with the counts are finite, and an ordinary column beside it."""
    n, m = 300, 260
    rows, _, dec = make_case(n, m, seed=4)
    rng = np.random.default_rng(2)
    gm = orc.genotype_mean(orc.popcounts(dec), n)
    x = dec.astype(np.float64) - gm[:, None].astype(np.float64)
    if which == "matvec":
        x = x.T
    v = rng.standard_normal((x.shape[1], 2)).astype(np.float32)
    v[:, 0] = 0
    v[5, 0] = size
    with api.Genotypes(rows, n) as g:
        g.set_weights(gm, np.ones(m, np.float32))
        got = getattr(g, which)(v)
    want = x @ v.astype(np.float64)
    assert np.all(np.linalg.norm(got - want, axis=0) <= 2e-6 * np.linalg.norm(want, axis=0))


def test_odd_sums_just_below_their_bound(gpu):
    """2^19 SNPs, one partial sum of each digit: the leading digits' sums of most individuals are odd integers
    between 2^24 − 2^11 and 2^24, which 24 bits just hold."""
    n, m = 130, 1 << 19
    odd = np.arange(64) * 8192 + 77                      # SNPs whose counts vary, with odd leading digits
    rng = np.random.default_rng(8)
    counts = np.full((odd.size, n), 2, np.uint8)
    counts[:] = rng.integers(0, 3, counts.shape)
    rows = np.full((m, (n + 3) // 4), 0xFF, np.uint8)    # every other count is 2
    rows[odd] = synth.encode_bed(counts)
    digit = np.full(m, 16.0)
    digit[odd] = rng.choice([7.0, 9.0, 11.0, 13.0], odd.size)
    sign = -1.0                                          # −16 is a digit, 16 the one above 15.5
    alpha = sign * (digit - np.where(digit == 16, 2.0 ** -30 * rng.integers(1, 2 ** 29, m), 0.0))
    with api.Genotypes(rows, n) as g:
        got = g.gebv(alpha)
    lead = (np.rint(-alpha)[odd][:, None] * counts).sum(0) + 2.0 * 16 * (m - odd.size)
    assert lead.max() <= 2 ** 24 and lead.min() >= 2 ** 24 - 2 ** 11 and (lead % 2 == 1).sum() > n // 4
    # effects in units of 2^-30: whole numbers, summed exactly
    a = np.rint(alpha * 2.0 ** 30).astype(np.int64)
    assert np.array_equal(a / 2.0 ** 30, alpha)
    rest = np.ones(m, bool)
    rest[odd] = False
    total = (a[odd][:, None] * counts.astype(np.int64)).sum(0) + 2 * int(a[rest].sum())
    assert np.array_equal(got, total.astype(np.longdouble).astype(np.float64) / 2.0 ** 30)


def test_long_digit_sums_are_split(gpu):
    """More than 2^19 K-elements, whose digit sums pass 2^24 in one accumulator."""
    n, m = 130, 690000
    rng = np.random.default_rng(6)
    rows = np.bitwise_or.reduce([rng.integers(0, 256, (m, (n + 3) // 4), dtype=np.uint8) for _ in range(3)])
    u = rng.uniform(0.96, 0.999, (m, 1)).astype(np.float32)
    want = np.zeros(n)
    for j in range(0, m, 50000):
        want += orc.bed_decode(rows[j:j + 50000], n).T.astype(np.float64) @ u[j:j + 50000, 0].astype(np.float64)
    assert want.min() * 16 > 2 ** 24
    with api.Genotypes(rows, n) as g:
        g.set_weights(np.zeros(m, np.float32), np.ones(m, np.float32))
        got = g.matvec(u)[:, 0]
    # 2^-24 of the largest value per entry, the digits' combination and the FP32 result
    assert np.all(np.abs(got - want) <= 2.0 ** -22 * want)
