"""The allocation-free field update at the edges of its paths: one to five types
(four is the last with 16-byte loads), cell counts that are and are not a multiple
of four, one tile and many, the sizes at which the tile grows, and buffers off a
16-byte boundary.  omega within 1e-6 of the FP64 expression, nothing written
outside, the energy the sum of its own omega times counts."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _omega64(n, scaling, xn, nref, literal):
    types = n.shape[0]
    phi = n.astype(np.float64) * scaling
    tot = phi.sum(axis=0)
    out = np.empty_like(phi)
    for t in range(types):
        w = (tot - 1.0) * xn[t, t] / nref
        for u in range(types):
            if u != t:
                w = w + (xn[u, t] * phi[u] if literal else -0.5 * xn[u, t] * (phi[t] - phi[u])) / nref
        out[t] = w
    return out


@pytest.mark.parametrize("literal", [0, 1])
@pytest.mark.parametrize("types", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("cells,shift", [(1, 0), (3, 0), (4, 0), (1000, 0), (1024, 0), (1028, 1), (4099, 0), (4100, 0),
                                         (2048 * 1024, 0), (2048 * 1024 + 4, 0), (2048 * 1024 + 4, 2)])
def test_noalloc_edges(types, cells, shift, literal):
    if cells > 10_000 and (types not in (2, 5) or literal):
        pytest.skip("the large sizes with two and five types are enough")
    import torch
    from new_arch_b200 import _lib
    rng = np.random.default_rng(cells + types)
    n = rng.poisson(24.0 / types, (types, cells)).astype(np.uint32)
    xn = rng.uniform(5.0, 50.0, (types, types))
    xn = xn + xn.T
    size = types * cells
    counts = torch.zeros(size + 8, dtype=torch.int32, device="cuda")
    counts[shift:shift + size] = torch.from_numpy(n.view(np.int32).reshape(-1)).cuda()
    omega = torch.full((size + 8,), 7.0, dtype=torch.float32, device="cuda")
    energy = torch.zeros(1, dtype=torch.float64, device="cuda")
    flat = np.ascontiguousarray(xn, dtype=np.float64)
    for _ in range(2):
        _lib.check(_lib.lib().scmf_update_omega_noalloc(
            counts.data_ptr() + 4 * shift, omega.data_ptr() + 4 * shift, types, cells, 1.0 / 24.0,
            flat.ctypes.data_as(C.POINTER(C.c_double)), 32, literal, energy.data_ptr(),
            torch.cuda.current_stream().cuda_stream))
    got = omega.cpu().numpy()
    assert (got[:shift] == 7.0).all() and (got[shift + size:] == 7.0).all()
    w = got[shift:shift + size].reshape(types, cells)
    want = _omega64(n, 1.0 / 24.0, xn, 32, literal)
    assert np.abs(w - want).max() <= 1e-6 * max(1.0, np.abs(want).max())
    e = float((w.astype(np.float64) * n).sum())
    assert abs(energy.item() - e) <= 1e-12 * max(1.0, np.abs(w.astype(np.float64) * n).sum())


def test_noalloc_in_a_callers_capture():
    """The call is made in someone else's stream capture and replayed there."""
    import torch
    from new_arch_b200 import _lib
    types, cells = 2, 5000
    counts = torch.randint(0, 30, (types * cells,), dtype=torch.int32, device="cuda")
    omega = torch.zeros(types * cells, dtype=torch.float32, device="cuda")
    energy = torch.zeros(1, dtype=torch.float64, device="cuda")
    xn = np.array([50.0, 20.0, 20.0, 50.0])

    def call():
        _lib.check(_lib.lib().scmf_update_omega_noalloc(
            counts.data_ptr(), omega.data_ptr(), types, cells, 1.0 / 24.0, xn.ctypes.data_as(C.POINTER(C.c_double)), 32, 0,
            energy.data_ptr(), torch.cuda.current_stream().cuda_stream))

    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    counts.copy_(torch.randint(0, 30, (types * cells,), dtype=torch.int32, device="cuda"))
    g.replay()
    torch.cuda.synchronize()
    got_w, got_e = omega.clone(), energy.item()
    call()
    torch.cuda.synchronize()
    assert torch.equal(omega, got_w) and energy.item() == got_e
