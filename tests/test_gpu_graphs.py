"""Bond graphs that are no linear chains on warp tiles: stars of five to seven arms
(seven bonds are one more than the tiles take), rings of two and three colours, beads
without a bond beside bonded ones, complete graphs of many colours, combs of the
longest chain of a tile and one bead more, one chain and several tiles a warp, linear
chains beside them, with and without the screen.  Positions and counts bit for bit
against the oracle."""
import os

import pytest

from tests._util import compare_state, oracle_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nb():
    import new_arch_b200
    return new_arch_b200


def _spec(nb, archs, smc_a, seed=5, grid=(12, 8, 10), count_bits=32):
    from new_arch_b200.spec import SystemSpec, cell_units, interaction_matrix
    return SystemSpec(2, *grid, *map(float, grid), interaction_matrix(2, 18.0, 50.0), 32, cell_units()[0], smc_a, seed,
                      nb.HAM_SCMF0, nb.FIELD_EVERY, count_bits, archs)


def _arch(length, chains, bonds):
    from new_arch_b200.spec import Arch, cell_units
    return Arch(length, chains, [(i // 3) % 2 for i in range(length)], [list(b) for b in bonds], cell_units()[1])


def _star(arms):
    return 1 + arms, [(0, i + 1) for i in range(arms)]


def _ring(n):
    return n, [(i, (i + 1) % n) for i in range(n)]


def _complete(n):
    return n, [(i, j) for i in range(n) for j in range(i)]


def _comb(length):
    """Every third backbone bead has a side bead; the side beads come last."""
    backbone = length - length // 4
    bonds = [(i, i + 1) for i in range(backbone - 1)]
    return length, bonds + [(3 * i, backbone + i) for i in range(length // 4)]


def _check(nb, spec, sweeps, what):
    with nb.System(spec) as s:
        s.init_coords()
        orc = oracle_for(spec)
        for n in sweeps:
            s.step(n)
            orc.step(n)
        compare_state(s, orc, what)
        assert s.validate()["ok"]


GRAPHS = {"star 5": _star(5), "star 6": _star(6), "star 7": _star(7), "ring 3": _ring(3), "ring 4": _ring(4),
          "ring 33": _ring(33), "loose": (7, [(1, 4), (4, 2)]), "loose 65": (65, [(1, 4)]), "star 66": (67, [(i // 5, i) for i in range(1, 67)]), "complete 6": _complete(6), "complete 7": _complete(7),
          "comb 40": _comb(40), "comb 1279": _comb(1279), "comb 1280": _comb(1280), "comb 1281": _comb(1281)}


@pytest.mark.parametrize("smc_a", [0.5, 0.02])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_graphs(nb, name, smc_a):
    length, bonds = GRAPHS[name]
    _check(nb, _spec(nb, [_arch(length, max(3, 6000 // length), bonds)], smc_a), (1, 4), f"{name}, A {smc_a}")


@pytest.mark.parametrize("smc_a", [0.5, 0.02])
def test_beside_linear_chains(nb, smc_a):
    from new_arch_b200.spec import linear_bonds
    archs = [_arch(33, 7, linear_bonds(33)), _arch(*_insert(_comb(41), 37)), _arch(32, 30, linear_bonds(32)),
             _arch(*_insert(_star(5), 101)), _arch(*_insert(_ring(9), 55))]
    _check(nb, _spec(nb, archs, smc_a, count_bits=16), (3,), f"beside linear chains, A {smc_a}")


def _insert(graph, chains):
    return graph[0], chains, graph[1]


def test_several_tiles_a_warp(nb):
    from oracle.oracle import set_threads
    set_threads(os.cpu_count() or 1)
    try:
        spec = _spec(nb, [_arch(*_insert(_comb(40), 150_000))], 0.5, grid=(64, 64, 64))
        _check(nb, spec, (2,), "several tiles")
    finally:
        set_threads(1)


def test_batch(nb):
    from new_arch_b200.spec import diblock_melt
    specs = [_spec(nb, [_arch(*_insert(_comb(40), 60))], 0.5, seed=3),
             diblock_melt(200, 33, 0.5, (10, 9, 8), 20.0, 50.0, seed=6, smc_a=0.02),
             _spec(nb, [_arch(*_insert(_ring(7), 90))], 0.02, seed=(7 << 40) + 1),
             _spec(nb, [_arch(*_insert(_star(4), 90))], 0.5, seed=9)]
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
