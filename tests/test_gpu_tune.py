"""What an autotune tries: one tuning where the batch runs many sweeps a launch, which no
option changes, the field tiles where its sweeps are launched one by one, and the move's
too where the general move kernel runs (a bead of seven bonds).  That kernel with several
tunings, bit for bit against the oracle."""
import pytest

from tests._util import compare_state, oracle_for

pytestmark = pytest.mark.gpu


def _star(arms, chains, seed, grid=(12, 10, 8)):
    import new_arch_b200 as nb
    from new_arch_b200.spec import Arch, SystemSpec, cell_units, interaction_matrix
    arch = Arch(1 + arms, chains, [i % 2 for i in range(1 + arms)], [[0, i + 1] for i in range(arms)], cell_units()[1])
    return SystemSpec(2, *grid, *map(float, grid), interaction_matrix(2, 18.0, 50.0), 32, cell_units()[0], 0.5, seed, nb.HAM_SCMF0,
                      nb.FIELD_EVERY, 32, [arch])


def _batch(specs, tune=None):
    import new_arch_b200 as nb
    systems = [nb.System(sp) for sp in specs]
    for s in systems:
        s.init_coords()
    return systems, nb.Batch(systems, tune=tune)


def _close(systems, b):
    b.close()
    for s in systems:
        s.close()


def test_trials():
    from new_arch_b200.spec import diblock_melt
    large = [diblock_melt(45_000, 32, 0.5, (64, 64, 40), 20.0, 50.0, seed=i) for i in range(2)]
    for specs, fields, moves in (([_star(4, 700, 3), _star(6, 300, 4)], {0}, 1), (large, {0, 2048, 8192, 32768}, 1),
                                 ([_star(7, 700, 3)], {0, 2048, 8192, 32768}, 24)):
        systems, b = _batch(specs)
        tune = b.autotune(2)
        trials = b.tune_trials()
        assert len(trials) == moves + len(fields) - 1
        assert {t["cells_per_tile"] for t in trials} == fields
        assert len({(t["beads_per_tile"], t["threads_move"], t["persistent_ctas"]) for t in trials}) == moves
        assert tune in [{k: v for k, v in t.items() if k in tune} for t in trials]
        _close(systems, b)


@pytest.mark.parametrize("tune", [{"chains_per_tile": 7, "threads_move": 64}, {"beads_per_tile": 1024, "threads_move": 256},
                                  {"chains_per_tile": 48, "persistent_ctas": 3}, {"use_graph": 0, "cells_per_tile": 100}])
def test_general_kernel(tune):
    specs = [_star(7, 300, 5), _star(8, 211, 6, (9, 8, 7)), _star(3, 100, 7)]
    systems, b = _batch(specs, tune)
    for n in (1, 4):
        b.step(n)
    for sp, s in zip(specs, systems):
        orc = oracle_for(sp)
        orc.step(5)
        compare_state(s, orc, f"seed {sp.seed}, {tune}")
    _close(systems, b)
