"""k_sweep_warp at the sizes where its tiles change kind: chains of one to three
beads, lengths that divide a warp's row and that do not, odd ones, the longest of
a tile of either size and one bead more, architectures that start at an odd
bead, few and many tiles a warp, screened and unscreened systems.  Positions and
counts bit for bit against the oracle."""
import numpy as np
import pytest

from tests._util import compare_state, oracle_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nb():
    import new_arch_b200
    return new_arch_b200


def _check(nb, spec, sweeps, what):
    with nb.System(spec) as s:
        s.init_coords()
        orc = oracle_for(spec)
        for n in sweeps:
            s.step(n)
            orc.step(n)
        compare_state(s, orc, what)
        assert s.validate()["ok"]


@pytest.mark.parametrize("smc_a", [0.5, 0.02])
@pytest.mark.parametrize("length", [2, 3, 16, 20, 33, 63, 64, 65, 488, 976, 977, 1984, 1985])
def test_lengths(nb, length, smc_a):
    chains = max(3, 6000 // length)
    spec = nb.spec.diblock_melt(chains, length, 0.4, (12, 8, 10), 20.0, 50.0, seed=length, smc_a=smc_a)
    _check(nb, spec, (1, 4), f"length {length}, A {smc_a}")


@pytest.mark.parametrize("grid", [(16, 16, 16), (24, 48, 20), (300, 6, 7)])
def test_architectures_at_odd_beads(nb, grid):
    """Five architectures (more than one launch's constants hold on the old fast
    path), odd ones first, so that the others start at every offset from a
    16-byte boundary; the three folds."""
    from new_arch_b200.spec import SystemSpec, cell_units, diblock_arch, homopolymer_arch, interaction_matrix
    k, sig = cell_units()
    archs = [diblock_arch(33, 0.5, 7, sig), homopolymer_arch(32, 0, 41, sig), homopolymer_arch(1, 1, 2, sig),
             diblock_arch(48, 0.3, 29, sig), homopolymer_arch(64, 1, 31, sig)]
    spec = SystemSpec(2, *grid, *map(float, grid), interaction_matrix(2, 18.0, 50.0), 32, k, 0.5, 99, nb.HAM_SCMF0,
                      nb.FIELD_EVERY, 16, archs)
    _check(nb, spec, (3,), f"odd beads, grid {grid}")


def test_several_tiles_a_warp(nb):
    """Enough chains that every warp strides over six tiles of unequal size."""
    spec = nb.spec.diblock_melt(430_000, 32, 0.5, (64, 64, 64), 20.0, 50.0, seed=8)
    from oracle.oracle import set_threads
    import os
    set_threads(os.cpu_count() or 1)
    try:
        _check(nb, spec, (2,), "several tiles")
    finally:
        set_threads(1)


def test_batch_of_screened_and_unscreened_systems(nb):
    """One launch over systems with and without the screen, of different seeds
    (upper halves too), stepped past one system's reference-rule field skip."""
    from new_arch_b200.spec import diblock_melt
    specs = [diblock_melt(300, 16, 0.5, (8, 8, 8), 20.0, 50.0, seed=5),
             diblock_melt(200, 33, 0.5, (10, 9, 8), 20.0, 50.0, seed=6, smc_a=0.02),
             diblock_melt(250, 48, 0.3, (16, 8, 8), 20.0, 50.0, seed=(7 << 40) + 1, field_rule=nb.FIELD_REFERENCE)]
    systems = [nb.System(sp) for sp in specs]
    for s in systems:
        s.init_coords()
    b = nb.Batch(systems)
    b.step(11)
    for sp, s in zip(specs, systems):
        orc = oracle_for(sp)
        orc.step(11)
        compare_state(s, orc, f"seed {sp.seed}")
    b.close()
    for s in systems:
        s.close()


def test_moves_are_written_back(nb):
    """Only beads that move are written: positions before and after a sweep
    differ in exactly the accepted moves."""
    spec = nb.spec.diblock_melt(4000, 32, 0.5, (16, 16, 16), 20.0, 50.0, seed=3)
    with nb.System(spec) as s:
        s.init_coords()
        before = s.coords().copy()
        st = s.step_stats(1)
        moved = int((s.coords() != before).any(axis=1).sum())
        assert moved == st["last_accepts"] and 0 < moved < spec.n_beads // 20
        assert np.isfinite(s.coords()).all()
