"""The marker QC's FP32 Hardy–Weinberg p-values (double-float walk) against the FP64 exact test of the
same counts, from equilibrium to far outside it (where the FP64 walk serves) and at small counts."""
import numpy as np
import pytest

from slemm_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("midp", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 61, 5000, 100001])
def test_marker_qc_hwe_matches_fp64_walk(gpu, n, midp):
    rng = np.random.default_rng(n)
    rows = []
    for f in (0.0, 0.0003, 0.01, 0.2, 0.5, 0.93, 1.0):
        for inbreeding in (0.0, 0.002, -0.01, 0.02, 0.1, -0.3, 0.9):
            het = max(0.0, 2 * f * (1 - f) * (1 - inbreeding))
            hom2 = min(1.0, max(0.0, f - het / 2))
            k = rng.multinomial(n, [max(0.0, 1 - min(1.0, het) - hom2), min(1.0, het), hom2][:3] / np.sum(
                [max(0.0, 1 - min(1.0, het) - hom2), min(1.0, het), hom2]))
            rows.append(np.repeat(np.arange(3, dtype=np.uint8), k))
    counts = np.stack(rows)
    with api.Genotypes(synth.encode_bed(counts), n) as g:
        _, hwep = g.marker_qc(midp)
    want = api.hwe_exact((counts == 1).sum(1), (counts == 0).sum(1), (counts == 2).sum(1), midp)
    # 1,500 pair operations of 2^-45 each at most, then the FP32 rounding
    assert np.all(np.abs(hwep - want) <= 2.0 ** -23 * want + 1e-45)
