"""Non-finite input reaches the outputs it belongs to, and only those."""
import numpy as np
import pytest
import torch

from test_gpu_kernel_edges import _sym, _table

pytestmark = pytest.mark.gpu

LS = [0, 1, 2, 1, 0]


def _one_electron(cuda, xyz, Z):
    from segfault_py_gb300.fock import FockBuilder
    fb = FockBuilder(_table(LS, [2, 1, 3, 2, 1], 8, 1.5), device=cuda)
    out = fb.one_electron(xyz, Z)
    fb.close()
    return out


def _forces(cuda, xyz, Z):
    from segfault_py_gb300 import _lib
    from segfault_py_gb300.fock import FockBuilder, _ptr, _stream_ptr
    n = sum((l + 1) * (l + 2) // 2 for l in LS)
    fb = FockBuilder(_table(LS, [2, 1, 3, 2, 1], 8, 1.5), device=cuda)
    d = [torch.tensor(x, device=cuda) for x in (xyz, Z, _sym(n, 1), _sym(n, 2))]
    g = torch.zeros(3 * len(Z), dtype=torch.float64, device=cuda)
    _lib.check(_lib.lib().sf_grad_one_electron(fb.handle, _ptr(d[0]), _ptr(d[1]), len(Z), _ptr(d[2]), _ptr(d[3]),
                                               _ptr(g), _stream_ptr()))
    fb.close()
    return g


def _geometry():
    return np.random.default_rng(2).uniform(-1, 2, (7, 3)), np.arange(1.0, 8.0)


def test_position_of_a_nucleus(cuda):
    """A Boys argument that is not a number has no table row: V and the forces that it
    enters are not numbers, S and T as before."""
    xyz, Z = _geometry()
    S, T, _ = _one_electron(cuda, xyz, Z)
    xyz[5, 1] = float("nan")
    S2, T2, V2 = _one_electron(cuda, xyz, Z)
    assert torch.equal(S, S2) and torch.equal(T, T2)
    assert torch.isnan(V2).all()
    g = _forces(cuda, xyz, Z).view(7, 3)
    assert torch.isnan(g[:6]).all() and torch.isfinite(g[6]).all()   # the shells' centres are atoms 0 to 4


def test_charge_of_a_nucleus(cuda):
    """A charge that is not a number makes V and the forces that it enters not numbers; S and T do not depend on
    charges."""
    xyz, Z = _geometry()
    S, T, _ = _one_electron(cuda, xyz, Z)
    Z[5] = float("nan")
    S2, T2, V2 = _one_electron(cuda, xyz, Z)
    assert torch.equal(S, S2) and torch.equal(T, T2)
    assert torch.isnan(V2).all()
    g = _forces(cuda, xyz, Z).view(7, 3)
    assert torch.isnan(g[:6]).all() and torch.isfinite(g[6]).all()
