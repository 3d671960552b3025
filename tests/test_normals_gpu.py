"""MC-REML's normal samples drawn on the GPU: fits at sample counts around the blocks of the draws'
compaction against the FP64 oracle, whose samples are libstdc++'s own."""
import numpy as np
import pytest

from oracle import slemm_np as orc
from slemm_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,n_MC,seed", [(501, 304, 1, 0), (700, 901, 1, 3), (512, 512, 8, 11), (1201, 450, 30, 2)])
def test_mc_reml_draws_vs_oracle(gpu, n, m, n_MC, seed):
    counts, _ = synth.simulate_counts(n, m, seed=n)
    y, _, _ = synth.simulate_phenotype(counts, 0.5, n_causal=100, seed=n)
    X = np.column_stack([np.ones(n), np.random.default_rng(n).standard_normal(n)]).astype(np.float32)
    y = y.astype(np.float32)
    want = orc.LMC_REML(counts, None, X, y, np.ones(m, np.float32), seed=seed, n_MC=n_MC, dtype=np.float64)
    with api.Genotypes(synth.encode_bed(counts), n) as g:
        got = g.LMC_REML(None, X, y, np.ones(m, np.float32), seed=seed, n_MC=n_MC)
    # other samples would move h2 by 1/sqrt(n·n_MC) > 5e-3; rounding moves it by 1e-6
    assert abs(got["h2"] - want["h2"]) <= 1e-4
    assert np.linalg.norm(got["Py"] - want["Py"]) <= 1e-3 * np.linalg.norm(want["Py"])
