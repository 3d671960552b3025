"""MC-REML's criterion terms (combination, projection, norms, scalings) at row counts and covariate counts at the
edges of their kernels, against the FP64 oracle."""
import numpy as np
import pytest

from oracle import slemm_np as orc
from slemm_gb300 import _lib, api, synth

pytestmark = pytest.mark.gpu


# 16-row words, rows in groups of four (vector loads) or not, more covariates than one pass takes, and more
# columns than the widest clusters serve
@pytest.mark.parametrize("n,m,c,n_MC", [(1501, 701, 6, 3), (1500, 700, 1, 3), (1039, 1203, 4, 9), (2064, 640, 5, 7)])
def test_mc_reml_at_kernel_edges(gpu, n, m, c, n_MC):
    counts, _ = synth.simulate_counts(n, m, seed=n)
    y, _, _ = synth.simulate_phenotype(counts, 0.4, n_causal=100, seed=2)
    rng = np.random.default_rng(n)
    X = np.column_stack([np.ones(n)] + [rng.standard_normal(n) for _ in range(c - 1)]).astype(np.float32)
    rvec = rng.uniform(0.5, 2.0, n).astype(np.float32)
    ps = np.ones(m, np.float32)
    y = y.astype(np.float32)
    r64 = orc.LMC_REML(counts, rvec, X, y, ps, seed=5, n_MC=n_MC, dtype=np.float64)
    with api.Genotypes(synth.encode_bed(counts), n) as g:
        g.set_precision(_lib.PREC_FP16X2)
        r = g.LMC_REML(rvec, X, y, ps, seed=5, n_MC=n_MC)
    # the bounds of the driver's other parity tests
    assert abs(r["h2"] - r64["h2"]) <= 1e-4
    assert np.corrcoef(r["snp_blup"], r64["snp_blup"])[0, 1] >= 0.99999
    assert np.allclose(r["blue"], r64["blue"], rtol=2e-3, atol=2e-3)
