"""The GA engine's sort and niche counts at the edges of their blocks and registers."""
import numpy as np
import pytest

from flexaidds_gb300 import evaluator, prepare, system
from oracle import ga

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("genes", [1, 4, 19, 63, 65, 100])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 129])
def test_niche_counts_against_the_oracle(n, genes):
    """Distances around the sharing radius, on it exactly (whole numbers), and zero."""
    rng = np.random.default_rng(100 * n + genes)
    ic = rng.integers(-3, 4, (n, genes)).astype(np.float64)
    ic[n // 2:] += rng.normal(0.0, 0.5, (n - n // 2, genes))
    ic[: n // 4] = ic[0]
    # n additions of terms of at most 1, and a rounding or two in each
    tol = (n + 4) * 2.0 ** -52
    for sig in (1.0, 2.0, 2.5):
        for alpha in (1.0, 2.0):
            want = np.array(ga.niche_counts(ic, sig, alpha))
            got = evaluator.ga_niche_counts(ic, sig, alpha)
            assert np.all(np.abs(got - want) <= tol * np.maximum(1.0, want)), (sig, alpha)


@pytest.mark.parametrize("population", [2, 3, 31, 33, 511, 1023, 1025, 2048])
def test_population_stays_sorted(tiny_system, population):
    _, d = tiny_system
    ev = evaluator.GPUEvaluator(d, max_poses=2 * population)
    eng = evaluator.GAEngine(max_jobs=1)
    slot = eng.admit(eng.job(ev, population, 4, seed=population), ev)
    for _ in range(3):
        eng.step()
        genes, e = eng.read_population(slot, population)
        assert np.all(np.diff(e) >= 0.0)
        again = ev.eval_genes(genes)["evalue"]
        np.testing.assert_array_equal(again, e)
    eng.close()
    ev.close()
