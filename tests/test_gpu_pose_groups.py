"""How a launch's poses are grouped (warps per group, poses per block, refills, the large shape for
polyhedra past the compact one's capacities) changes no pose's record."""
import numpy as np
import pytest

from flexaidds_gb300 import evaluator, prepare, synth, system
from oracle import port

pytestmark = pytest.mark.gpu

SMS, WARPS, SPLIT = 152, 16, 4


@pytest.fixture(scope="module")
def poses():
    """More poses than the device scores at once, mostly scored ones, their records from one launch."""
    d = prepare.prepare(system.make_inputs(600, 6.0, 12, 3, seed=5, side_chains=1, rotamers=4))
    n = SMS * WARPS + 200
    pool = synth.random_genes(60000, d.n_genes, seed=6)
    ev = evaluator.GPUEvaluator(d, max_poses=4096)
    ok = pool[ev.eval_genes(pool)["status"] == 0]
    rng = np.random.default_rng(1)
    genes = np.ascontiguousarray(np.concatenate([ok[rng.integers(0, len(ok), n - 300)], pool[:300]])[rng.permutation(n)])
    yield ev, genes, ev.eval_genes(genes).copy()
    ev.close()


@pytest.mark.parametrize("n", [1, 2, 3, SMS - 1, SMS, SMS + 1, 2 * SMS + 1, SPLIT * SMS, SPLIT * SMS + 1,
                               WARPS * SMS - 1, WARPS * SMS, WARPS * SMS + 1])
def test_records_do_not_depend_on_the_launch(poses, n):
    ev, genes, all_records = poses
    at = np.random.default_rng(n).permutation(len(genes))[:n]
    np.testing.assert_array_equal(ev.eval_genes(np.ascontiguousarray(genes[at])), all_records[at])


@pytest.mark.parametrize("shell,radius,atom", [(52, 5.2, 2.0), (62, 4.4, 2.0), (62, 5.6, 1.4), (70, 5.2, 2.0), (84, 4.8, 2.0),
                                              (84, 5.6, 2.0)])
def test_polyhedra_past_the_compact_shape(shell, radius, atom):
    """Ligands inside a shell of receptor atoms all about as far away: cells with far more faces than a
    packing of atoms gives (past the compact shape's vertices, points or items in none to nearly all of the
    poses, some past the 200 hull edges too), against the oracle."""
    base = system.make_inputs(600, 6.0, 12, 3, seed=5)
    k = np.arange(shell) + 0.5
    phi, z = np.pi * (1.0 + 5.0 ** 0.5) * k, 1.0 - 2.0 * k / shell
    r = np.sqrt(1.0 - z * z)
    xyz = radius * np.stack([r * np.cos(phi), r * np.sin(phi), z], axis=1)
    xyz += np.random.default_rng(shell).normal(0.0, 0.05, xyz.shape)
    far = base.receptor.xyz - base.receptor.cleft_center
    xyz = np.concatenate([xyz, far[np.linalg.norm(far, axis=1) > 9.5]]).astype(np.float32)
    n = len(xyz)
    rec = synth.Receptor(xyz=xyz, type=np.resize(base.receptor.type, n), radius=np.full(n, atom, np.float32),
                         cleft_center=np.zeros(3, np.float32), cleft_radius=2.0, edge=12.0)
    grid = np.random.default_rng(2).uniform(-0.3, 0.3, (200, 3)).astype(np.float32)
    d = prepare.prepare(system.SystemInputs(receptor=rec, ligand=synth.random_ligand(4, 0, seed=3), grid_xyz=grid,
                                            emat=base.emat))
    genes = synth.random_genes(1500, d.n_genes, seed=4)
    port.set_reference_compat(True)
    port.set_trig_rounding(False)
    want = port.Oracle(d).eval_ic(d.genes_to_ic(genes))["cf"]
    ev = evaluator.GPUEvaluator(d, max_poses=2048)
    got = ev.eval_genes(genes)
    assert ev.stats()["capacity"] == 0
    ev.close()
    np.testing.assert_array_equal(got["status"], want["status"])
    assert (want["status"] != 2).sum() >= 50
    err = np.abs(got["evalue"] - want["evalue"]) / np.maximum(1.0, np.abs(want["evalue"]))
    assert err.max() <= 1e-9
