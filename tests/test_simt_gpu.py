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
