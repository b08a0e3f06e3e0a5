"""The launch of many sweeps with any omega: sweep 10 keeps the caller's (the reference
rule), with a span that is unknown, wide or none, the sweeps after it use new ones.
Positions, counts and accepted moves after every call bit for bit against the oracle."""
import numpy as np
import pytest

from tests._util import assert_coords_equal, assert_counts_equal, oracle_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,smc_a", [(32, 0.5), (33, 0.5), (80, 0.5), (32, 0.02)])
@pytest.mark.parametrize("values", [[40.0, -40.0], [np.nan], [np.inf, -np.inf]])
def test_any_omega(length, smc_a, values):
    import new_arch_b200 as nb
    from new_arch_b200.spec import diblock_melt
    spec = diblock_melt(round(7.8 * 16 ** 3 / length), length, 0.3, (16, 16, 16), 25.0, 50.0, seed=21, smc_a=smc_a,
                        field_rule=nb.FIELD_REFERENCE)
    rng = np.random.default_rng(3)
    with nb.System(spec) as s:
        s.init_coords()
        orc = oracle_for(spec)
        s.step(3)
        orc.step(3)
        for first in (9, 8, 18):  # steps before the calls below
            for x in (s, orc):
                x.set_step(first)
            w = s.omega().copy()
            at = rng.choice(w.size, size=w.size // 50, replace=False)
            w[at] = rng.choice(np.float32(values), at.size)
            for x in (s, orc):
                x.set_omega(w)
            for n in (2, 5):
                s.step(n)
                orc.step(n)
                what = f"{length}, {values}, {n} sweeps from {first}"
                assert_coords_equal(s.coords(), orc.coords(), what)
                assert_counts_equal(s.counts(), orc.counts(), what)
                assert s.sweep_stats()["total_accepts"] == orc.stats()["total_accepts"], what
