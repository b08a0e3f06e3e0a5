"""Few chains on large grids, whose sweeps are launched one by one, on either side of the
cells a launch of many sweeps takes: two and four types, cells that do not come in fours,
a branched chain, a batch with a system that would fit alone.  Positions and counts bit
for bit against the oracle."""
import pytest

from tests._util import compare_state, oracle_for

pytestmark = pytest.mark.gpu


def _spec(chains, grid, types=2, bonds=None, length=32, seed=4, rule=None):
    import new_arch_b200 as nb
    from new_arch_b200.spec import Arch, SystemSpec, cell_units, interaction_matrix, linear_bonds
    arch = Arch(length, chains, [i * types // length for i in range(length)], bonds or linear_bonds(length), cell_units()[1])
    return SystemSpec(types, *grid, *map(float, grid), interaction_matrix(types, 18.0, 50.0), 32, cell_units()[0], 0.5, seed,
                      nb.HAM_SCMF0, nb.FIELD_EVERY if rule is None else rule, 32, [arch])


def _check(spec, s, orc, what):
    for n in (2, 9):
        s.step(n)
        orc.step(n)
    compare_state(s, orc, what)
    assert s.validate()["ok"]


@pytest.mark.parametrize("chains,grid,types", [(1, (12, 8, 4), 2), (1, (12, 8, 24), 2), (5, (16, 18, 16), 2), (5, (24, 24, 24), 2),
                                               (40, (47, 31, 29), 2), (40, (16, 16, 30), 4), (40, (32, 24, 20), 4)])
def test_grids(chains, grid, types):
    import new_arch_b200 as nb
    spec = _spec(chains, grid, types)
    with nb.System(spec) as s:
        s.init_coords()
        _check(spec, s, oracle_for(spec), f"{chains} chains on {grid}, {types} types")


def test_ring():
    import new_arch_b200 as nb
    spec = _spec(9, (40, 40, 20), bonds=[[i, (i + 1) % 33] for i in range(33)], length=33, rule=nb.FIELD_REFERENCE)
    with nb.System(spec) as s:
        s.init_coords()
        _check(spec, s, oracle_for(spec), "rings")


def test_batch():
    import new_arch_b200 as nb
    specs = [_spec(60, (8, 8, 8), seed=5), _spec(3, (40, 30, 41), seed=6)]
    systems = [nb.System(sp) for sp in specs]
    for s in systems:
        s.init_coords()
    b = nb.Batch(systems)
    b.step(2)
    b.step(9)
    for sp, s in zip(specs, systems):
        orc = oracle_for(sp)
        orc.step(11)
        compare_state(s, orc, f"seed {sp.seed}")
    b.close()
    for s in systems:
        s.close()
