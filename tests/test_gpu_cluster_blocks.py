"""Clustering at the edges of the build's and the passes' blocks and of the atoms a pass loads at a time,
against the oracle."""
import numpy as np
import pytest

from flexaidds_gb300 import evaluator, prepare, synth, system
from test_cluster import assert_same, oracle_cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms", [4, 5, 13])
def test_cluster_block_edges(atoms):
    d = prepare.prepare(system.make_inputs(600, 6.0, atoms, 1, seed=5))
    ic, e = synth.clustered_ensemble(d, 8, 70, seed=atoms)
    rng = np.random.default_rng(atoms)
    ev = evaluator.GPUEvaluator(d, max_poses=64)
    for n in (1, 2, 127, 128, 129, 255, 257, 513):
        at = np.sort(rng.permutation(len(e))[:n])
        for T, R in ((0, 5), (300, 12)):
            i, x = np.ascontiguousarray(ic[at]), np.ascontiguousarray(e[at])
            assert_same(ev.cluster(i, x, T, 1.0, R), oracle_cluster(d, i, x, T, 1.0, R), R)
    ev.close()
