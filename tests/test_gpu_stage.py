"""Large host copies: sizes on both sides of the line from which a copy goes through
the pinned buffer, a last piece of one bead, page-locked memory, and two systems that
copy at once (one of them takes the driver's copy).  Bytes as set, and the grid that of
those positions."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_LINE = 64 << 20


@pytest.fixture(scope="module")
def nb():
    import new_arch_b200
    return new_arch_b200


def _system(nb, beads):
    from new_arch_b200.spec import SystemSpec, cell_units, homopolymer_arch, interaction_matrix
    k, sig = cell_units()
    return nb.System(SystemSpec(1, 32, 32, 32, 32.0, 32.0, 32.0, interaction_matrix(1, 0.0, 50.0), 32, k, 0.5, 3,
                                nb.HAM_SCMF0, nb.FIELD_EVERY, 32, [homopolymer_arch(1, 0, beads, sig)]))


def _positions(beads, seed):
    return np.random.default_rng(seed).uniform(0.0, 32.0, (beads, 3)).astype(np.float32)


def _counts(x):
    c = np.floor(x).astype(np.int64) % 32
    return np.bincount(c[:, 0] + 32 * (c[:, 1] + 32 * c[:, 2]), minlength=32 ** 3)


@pytest.mark.parametrize("beads", [_LINE // 12, _LINE // 12 + 1, (_LINE + (9 << 20)) // 12 + 1, 7_000_003])
def test_round_trip(nb, beads):
    x = _positions(beads, beads)
    with _system(nb, beads) as s:
        s.set_coords(x)
        assert np.array_equal(s.coords(), x)
        assert np.array_equal(s.counts(), _counts(x))


def test_page_locked(nb):
    import torch
    from new_arch_b200 import _lib
    beads = 6_000_001
    x = torch.from_numpy(_positions(beads, 1)).pin_memory()
    out = torch.empty_like(x).pin_memory()
    with _system(nb, beads) as s:
        s.set_coords(x.numpy())
        _lib.check(_lib.lib().scmf_get_coords(s._h, C.cast(out.data_ptr(), C.POINTER(C.c_float)), out.numel()))
    assert torch.equal(x, out)


def test_two_at_once(nb):
    beads, errors = 8_000_001, []

    def work(seed):
        try:
            for i in range(3):
                x = _positions(beads, 10 * seed + i)
                with _system(nb, beads) as s:
                    s.set_coords(x)
                    assert np.array_equal(s.coords(), x)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
