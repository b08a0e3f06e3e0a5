"""The screen of the linear-chain move kernel (k_sweep_warp), on the CPU: its
piecewise-linear normals stay within the error the screen allows for, and a
trial that its inequality rejects is one that the exact trial rejects whatever
omega holds (to within the span)."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "new_arch_b200", "csrc")


def _table(name, cols):
    text = open(os.path.join(CSRC, name)).read()
    body = text[text.index("TABLE_DATA"):]
    vals = [float.fromhex(v[:-1]) if "x" in v else float(v[:-1]) for v in re.findall(r"-?[0-9][0-9a-fx.p+-]*f", body)]
    return np.array(vals, dtype=np.float32).reshape(-1, cols)


EXACT, SCREEN = _table("scmf_normal_table.h", 4), _table("scmf_screen_table.h", 2)
DELTA = float(re.search(r"SCREEN_DELTA (\S+)", open(os.path.join(CSRC, "scmf_screen_table.h")).read()).group(1))


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


def _float_of(w):
    return ((w.astype(np.uint64) << np.uint64(1)) & np.uint64(0xFFFFFFFF) | np.uint64(1)).astype(np.float32)


def exact_normal(w):
    bits = _float_of(w).view(np.uint32)
    c = EXACT[(bits >> 19) - (127 << 4)]
    t = ((bits & 0x7FFFF) | 0x3F800000).view(np.float32) - np.float32(1.03125)
    z = _fma(_fma(_fma(c[:, 3], t, c[:, 2]), t, c[:, 1]), t, c[:, 0])
    return np.where(w >> 31, -z, z)


def screen_normal(w):
    f = _float_of(w)
    c = SCREEN[(f.view(np.uint32) >> 21) - (127 << 2)]
    z = _fma(c[:, 1], f, c[:, 0])
    return np.where(w >> 31, -z, z).astype(np.float64) * 2.0 ** -30


def _words(seed):
    rng = np.random.default_rng(seed)
    # every binade alike, the ends of the range, and the edges of the segments
    spread = (2.0 ** rng.uniform(0, 31, 2_000_000)).astype(np.uint64)
    edges = np.concatenate([np.uint64(2) ** np.uint64(e) * np.arange(4, 8, dtype=np.uint64) // np.uint64(4) for e in range(31)])
    w = np.concatenate([spread, edges, edges + np.uint64(1), np.maximum(edges, np.uint64(1)) - np.uint64(1),
                        np.array([0, 1, 2**31 - 1, 2**31 - 2], np.uint64), rng.integers(0, 2**32, 1_000_000, dtype=np.uint64)])
    return np.concatenate([w, w ^ np.uint64(1 << 31)]).astype(np.uint32)


def test_screen_normals_within_their_bound():
    assert SCREEN.shape[0] == 129 and EXACT.shape[0] == 513
    w = _words(1)
    worst = np.abs(screen_normal(w) - exact_normal(w)).max()
    assert worst <= DELTA, worst


@pytest.mark.parametrize("A,k", [(0.5, 3.0 / 0.98), (0.5, 30.0), (2.0, 3.0), (0.04, 46.5)])
@pytest.mark.parametrize("deg", [1, 2])
def test_screened_trials_are_rejected_whatever_omega(A, k, deg):
    """The inequality of ScreenDev in the kernel's own FP32 steps, against the
    exact energy in FP32: dE_bond >= span - log u for every screened trial."""
    rng = np.random.default_rng(7)
    n = 400_000
    f4 = np.float32
    A, R, c = f4(A), f4(np.sqrt(2.0 * A)), f4(2 * k) * f4(deg)
    ac4 = (A * c) * f4(0.25)
    span = rng.choice(np.array([0.0, 1e-3, 0.5, 3.0, 40.0], f4), n)
    # forces from none to far beyond equilibrium (sigma sqrt(c))
    f = (rng.standard_normal((n, 3)) * np.sqrt(float(c)) * 2.0 ** rng.uniform(-6, 6, (n, 1))).astype(f4)
    w = rng.integers(0, 2**32, (n, 4), dtype=np.uint64).astype(np.uint32)
    # as the kernel screens
    eta, unit = 2.0 ** -6, 2.0 ** 30
    up = lambda v: np.nextafter(f4(v), f4(np.inf))  # noqa: E731
    K = (1 + eta) * (1 + 2.0 ** -10)
    a = f4((float(A) - 1.0 / float(c)) / float(R) * unit)
    b = up(K / (float(c) * float(R)) ** 2 * unit * unit)
    add = up((1 + 1 / eta) * 3 * DELTA * DELTA * unit * unit)
    four = up(4.0 / float(A))
    u0, u1 = four * (span + f4(2.0 ** -18)), four * f4(-float.fromhex("0x1.62e7p-1"))
    v = [_fma(f[:, i], np.full(n, a), (screen_normal(w[:, i]) * unit).astype(f4)) for i in range(3)]
    q = _fma(v[0], v[0], _fma(v[1], v[1], v[2] * v[2]))
    below = _fma(w[:, 3].astype(f4), np.full(n, f4(-2.0 ** -32)), np.full(n, f4(1 - 2.0 ** -23)))
    with np.errstate(divide="ignore", invalid="ignore"):
        lg = np.log2(below.astype(np.float64)).astype(f4)
    lim = _fma(np.full(n, b), _fma(f[:, 0], f[:, 0], _fma(f[:, 1], f[:, 1], _fma(f[:, 2], f[:, 2], _fma(lg, np.full(n, u1), u0)))),
               np.full(n, add))
    screened = q > lim
    # the exact trial
    d = [_fma(np.full(n, A), f[:, i], R * exact_normal(w[:, i]).astype(f4)) for i in range(3)]
    d2 = _fma(d[0], d[0], _fma(d[1], d[1], d[2] * d[2]))
    fd = _fma(f[:, 0], d[0], _fma(f[:, 1], d[1], f[:, 2] * d[2]))
    deb = ac4 * _fma(np.full(n, c), d2, f4(-2.0) * fd)
    u = f4(2.0) - ((w[:, 3] >> 9) | np.uint32(0x3F800000)).view(f4)
    lowest = deb.astype(np.float64) - span          # of dE, over all omega
    may_pass = lowest < -np.log(u.astype(np.float64))
    assert not (screened & may_pass).any()
    assert screened.any() and (~screened).any()
    if float(A) * 4 * k > 4 and deg == 2:           # and it does screen where it runs, at forces of equilibrium
        near = (np.abs(f) < 2 * np.sqrt(float(c))).all(axis=1) & (span < 1)
        assert screened[near].mean() > 0.8
