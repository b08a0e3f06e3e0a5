"""Short odd chains that fill their warp tiles: single beads beside combs and beside chains
of 1,200, trimers beside chains of 970, where a tile's bead pairs and not its beads are
what limits it, with and without the screen.  Every trial is made: positions and counts
bit for bit against the oracle."""
import os

import pytest

from tests._util import compare_state, oracle_for

pytestmark = pytest.mark.gpu


def _comb40():
    """A backbone of 24 with two-bead side chains at every third bead."""
    bonds, n = [[i, i + 1] for i in range(23)], 24
    for b in range(0, 24, 3):
        bonds += [[b, n], [n, n + 1]]
        n += 2
    return n, bonds


def _linear(length):
    return length, [[i, i + 1] for i in range(length - 1)]


MIXES = {"combs and single beads": ((_comb40(), 50_000), (_linear(1), 100_000)),
         "chains of 1,200 and single beads": ((_linear(1200), 1000), (_linear(1), 200_000)),
         "chains of 970 and trimers": ((_linear(970), 1200), (_linear(3), 350_000))}


@pytest.mark.parametrize("smc_a", [0.5, 0.02])
@pytest.mark.parametrize("name", sorted(MIXES))
def test_every_trial_is_made(name, smc_a):
    import new_arch_b200 as nb
    from new_arch_b200.spec import Arch, SystemSpec, cell_units, interaction_matrix
    from oracle.oracle import set_threads
    archs = [Arch(n, chains, [(i // 3) % 2 for i in range(n)], bonds, cell_units()[1]) for (n, bonds), chains in MIXES[name]]
    spec = SystemSpec(2, 64, 64, 60, 64.0, 64.0, 60.0, interaction_matrix(2, 18.0, 50.0), 32, cell_units()[0], smc_a, 11,
                      nb.HAM_SCMF0, nb.FIELD_EVERY, 32, archs)
    set_threads(os.cpu_count() or 1)
    try:
        with nb.System(spec) as s:
            s.init_coords()
            orc = oracle_for(spec)
            for n in (1, 2):
                s.step(n)
                orc.step(n)
            compare_state(s, orc, f"{name}, A {smc_a}")
    finally:
        set_threads(1)
