"""k_sweep_pairs: unscreened systems of more beads than the chip holds, of chains of up to
64 beads.  Even lengths on grids of the three folds, lengths that leave lanes of a row
without a pair, chains of one and three beads, architectures at odd beads, several in one
system, batches of several seeds and count widths, and moves without counts.  Positions
and counts bit for bit against the oracle."""
import os

import pytest

from tests._util import assert_coords_equal, compare_state, oracle_for

pytestmark = pytest.mark.gpu
BEADS = 2_600_000  # more tiles than warps in any form


@pytest.fixture(scope="module", autouse=True)
def oracle_threads():
    from oracle.oracle import set_threads
    set_threads(os.cpu_count() or 1)
    yield
    set_threads(1)


def _spec(archs, grid, seed=21, smc_a=0.02, count_bits=32):
    import new_arch_b200 as nb
    from new_arch_b200.spec import SystemSpec, cell_units, diblock_arch, interaction_matrix
    k, sig = cell_units()
    return SystemSpec(2, *grid, *map(float, grid), interaction_matrix(2, 18.0, 50.0), 32, k, smc_a, seed, nb.HAM_SCMF0,
                      nb.FIELD_EVERY, count_bits, [diblock_arch(n, 0.4, chains, sig) for n, chains in archs])


def _check(spec, what, sweeps=6):
    import new_arch_b200 as nb
    with nb.System(spec) as s:
        s.init_coords()
        orc = oracle_for(spec)
        s.step(sweeps)
        orc.step(sweeps)
        compare_state(s, orc, what)


@pytest.mark.parametrize("length,grid", [(2, (64, 64, 32)), (32, (64, 64, 64)), (64, (72, 60, 59)), (16, (300, 30, 31)),
                                         (48, (64, 64, 64)), (22, (40, 50, 60)), (20, (64, 64, 64)),
                                         (1, (64, 64, 64)), (3, (300, 30, 31)), (31, (72, 60, 59)), (49, (64, 64, 64))])
def test_lengths(length, grid):
    _check(_spec([(length, BEADS // length + 1)], grid), f"length {length} on {grid}")


@pytest.mark.parametrize("grid", [(64, 64, 64), (72, 60, 59)])
def test_architectures(grid):
    n = BEADS // 4
    even = [(32, n // 32 + 1), (64, n // 64 + 1), (8, n // 8 + 3), (48, n // 48 + 1)]
    _check(_spec(even, grid), f"even lengths on {grid}")
    _check(_spec([(3, 7)] + even, grid), f"odd beads on {grid}")


def test_branched_chains_beside(grid=(64, 64, 64)):
    """Not for k_sweep_pairs: the same sizes with a branched architecture, alone and beside linear chains."""
    from new_arch_b200.spec import Arch, cell_units
    star = Arch(5, BEADS // 10, [0, 1, 1, 0, 1], [[0, 1], [0, 2], [0, 3], [0, 4]], cell_units()[1])
    for archs in ([(32, BEADS // 64)], []):
        spec = _spec(archs, grid)
        spec.archs.append(star)
        _check(spec, f"stars beside {archs}")
    star.n_chains *= 2
    _check(spec, "stars")


def test_moves_without_counts():
    import new_arch_b200 as nb
    spec = _spec([(32, BEADS // 32)], (64, 64, 64))
    with nb.System(spec) as s:
        s.init_coords()
        orc = oracle_for(spec)
        before = s.counts()
        s.smc_move(1)
        assert (s.counts() == before).all()
        s.reset_density_fields()
        s.update_omega_fields_scmf0()
        orc.step(1)
        assert_coords_equal(s.coords(), orc.coords(), "smc_move")
        compare_state(s, orc, "smc_move", energies=False)


@pytest.mark.parametrize("length", [32, 3])
def test_any_omega(length):
    """The caller's omega with NaN, infinite and very large cells among ordinary ones."""
    import numpy as np
    import new_arch_b200 as nb
    spec = _spec([(length, BEADS // length + 1)], (64, 64, 64))
    with nb.System(spec) as s:
        s.init_coords()
        orc = oracle_for(spec)
        rng = np.random.default_rng(5)
        w = rng.normal(0.0, 2.0, 2 * 64 ** 3).astype(np.float32)
        odd = rng.integers(0, w.size, w.size // 20)
        w[odd] = rng.choice(np.float32([np.nan, np.inf, -np.inf, 3e38, -3e38, 1e-40, -0.0]), odd.size)
        s.set_omega(w)
        orc.set_omega(w)
        s.smc_move(2)
        orc.smc_move(2)
        assert_coords_equal(s.coords(), orc.coords(), "any omega")


@pytest.mark.parametrize("seeds", ["one", "upper half", "any"])
def test_batch(seeds):
    import new_arch_b200 as nb
    seed = {"one": lambda i: 9, "upper half": lambda i: (5 << 40) + i, "any": lambda i: (i << 40) + 3}[seeds]
    shapes = [((32, 40_000), (64, 48, 32), 32), ((48, 10_001), (40, 30, 20), 32), ((3, 200_001), (64, 32, 32), 32),
              ((16, 4001), (16, 16, 16), 16), ((64, 9000), (33, 32, 31), 32)]
    specs = [_spec([arch], grid, seed(i + 1), count_bits=bits) for i, (arch, grid, bits) in enumerate(shapes)]
    systems = [nb.System(sp) for sp in specs]
    for s in systems:
        s.init_coords()
    b = nb.Batch(systems)
    b.step(8)
    for sp, s in zip(specs, systems):
        orc = oracle_for(sp)
        orc.step(8)
        compare_state(s, orc, f"seed {sp.seed}")
    b.close()
    for s in systems:
        s.close()
