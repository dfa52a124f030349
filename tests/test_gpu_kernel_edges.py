"""Kernels at the sizes where their layouts change, against the oracle.

One-electron kernels: lanes per primitive pair follow the number of primitive
pairs (1, 2, more), lanes share nuclei (fewer, as many, more than lanes), and the
gradient keeps its forces in shared memory up to 128 nuclei.  Raw integrals: a
quartet goes to part of a warp, a CTA or a cluster by its primitive quartets.
Two-electron gradient: every class (work tables of one, some and 32 lanes).

Tolerances.  FP64 sums here have at most 5e3 terms, none larger than the largest
element by more than 10, each rounded to 1.1e-16: 5e-12 of the largest element.
Central differences with step 1e-4 bohr leave h^2/6 f''' <= 1.7e-9 x 1e2 for
exponents up to 3 plus 1e-14 / h of rounding: 1e-6 of the largest component.
FP32 derivative quartets: 6e-8 per operation, times 2 alpha |r| <= 50 and some
tens of operations: 1e-4."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle as O
from test_gpu_parity import _shell_cgfs

pytestmark = pytest.mark.gpu


def _table(ls, nprim, seed, box, emin=0.2, emax=3.0):
    """Random shells with the given l and contraction lengths, each its own atom."""
    rng = np.random.default_rng(seed)
    n = len(ls)
    nc = [(l + 1) * (l + 2) // 2 for l in ls]
    po = np.concatenate([[0], np.cumsum(nprim)]).astype(np.int32)
    return dict(l=np.array(ls, dtype=np.int32), nprim=np.array(nprim, dtype=np.int32),
                atom=np.arange(n, dtype=np.int32),
                ao_offset=np.concatenate([[0], np.cumsum(nc)[:-1]]).astype(np.int32),
                center=rng.uniform(0, box, (n, 3)), prim_offset=po,
                exps=np.exp(rng.uniform(np.log(emin), np.log(emax), po[-1])), coefs=rng.uniform(0.3, 1.0, po[-1]))


def _cgfs(table):
    return [c for s in range(len(table["l"])) for c in _shell_cgfs(table, s)]


def _sym(n, seed):
    A = np.random.default_rng(seed).standard_normal((n, n))
    return 0.5 * (A + A.T)


@pytest.mark.parametrize("natom", [1, 7, 8, 9, 33, 130])
@pytest.mark.parametrize("nprim", [1, 2, 3, 6])
def test_one_electron_layouts(cuda, nprim, natom):
    from segfault_py_gb300.fock import FockBuilder
    # contractions 1 and nprim together: pairs of 1, nprim and nprim^2 primitives
    table = _table([0, 1, 2, 0, 1, 2], [1, 1, 1, nprim, nprim, nprim], 3 + nprim, 3.0)
    rng = np.random.default_rng(natom)
    xyz, Z = rng.uniform(-2, 5, (natom, 3)), rng.integers(1, 9, natom).astype(np.float64)
    fb = FockBuilder(table, device=cuda)
    got = fb.one_electron(xyz, Z)
    for name, a, b in zip("STV", got, O.one_electron(_cgfs(table), xyz, Z)):
        assert np.abs(a.cpu().numpy() - b).max() <= 5e-12 * np.abs(b).max(), name
    fb.close()


@pytest.mark.parametrize("extra", [0, 140])
@pytest.mark.parametrize("nprim", [1, 3])
def test_one_electron_gradient_layouts(cuda, nprim, extra):
    """sf_grad_one_electron against central differences of sum D (T + V) - W S from the oracle; the shells'
    own atoms come first, `extra` charges follow (over 128 nuclei: forces straight to global memory)."""
    from segfault_py_gb300 import _lib
    from segfault_py_gb300.fock import FockBuilder, _ptr, _stream_ptr
    ls = [0, 1, 2, 1]
    table = _table(ls, [1, nprim, nprim, 2], 11, 2.5)
    rng = np.random.default_rng(5)
    n = sum((l + 1) * (l + 2) // 2 for l in ls)
    nuc = np.concatenate([table["center"], rng.uniform(-6, 9, (extra, 3))])
    Z = rng.integers(1, 5, len(nuc)).astype(np.float64)
    D, W = _sym(n, 1), _sym(n, 2)

    def energy(x):
        t = dict(table, center=x[:len(ls)])
        S, T, V = O.one_electron(_cgfs(t), x, Z)
        return np.sum(D * (T + V)) - np.sum(W * S)

    fb = FockBuilder(table, device=cuda)
    d = [torch.tensor(x, device=cuda) for x in (nuc, Z, D, W)]
    g = torch.zeros(3 * len(nuc), dtype=torch.float64, device=cuda)
    _lib.check(_lib.lib().sf_grad_one_electron(fb.handle, _ptr(d[0]), _ptr(d[1]), len(nuc), _ptr(d[2]), _ptr(d[3]),
                                               _ptr(g), _stream_ptr()))
    g = g.cpu().numpy().reshape(-1, 3)
    fb.close()
    assert np.abs(g.sum(axis=0)).max() <= 1e-9 * np.abs(g).max()
    for a, k in [(0, 0), (1, 1), (2, 2), (3, 0), (2, 1)] + ([(4, 2), (100, 0)] if extra else []):
        h = np.zeros_like(nuc)
        h[a, k] = 1e-4
        fd = (energy(nuc + h) - energy(nuc - h)) / 2e-4
        assert abs(fd - g[a, k]) <= 1e-6 * np.abs(g).max(), (a, k, fd, g[a, k])


@pytest.mark.parametrize("profiling", [0, 2])
@pytest.mark.parametrize("precision", ["fp64", "df"])
def test_gradient_parts_side_by_side(cuda, precision, profiling):
    """sf_grad_rhf adds what sf_grad_one_electron and sf_grad_jk add, in another order: fewer than 1e5
    terms of at most the largest force each in FP64 (double-float: 2^-44 each), 1e-11 of the largest."""
    from segfault_py_gb300 import _lib
    from segfault_py_gb300.fock import FockBuilder, _ptr, _stream_ptr
    ls = [0, 1, 2, 1, 0]
    table = _table(ls, [2, 1, 1, 3, 2], 4, 2.0)
    n = sum((l + 1) * (l + 2) // 2 for l in ls)
    L = _lib.lib()
    fb = FockBuilder(table, device=cuda, cutoff=0.0)
    d = [torch.tensor(x, device=cuda) for x in (table["center"], np.arange(1.0, 6.0), _sym(n, 1), _sym(n, 2))]
    p = [_ptr(x) for x in d]
    apart, both = (torch.ones(15, dtype=torch.float64, device=cuda) for _ in range(2))
    prec = _lib.PRECISION[precision]
    _lib.check(L.sf_grad_one_electron(fb.handle, p[0], p[1], 5, p[2], p[3], _ptr(apart), _stream_ptr()))
    _lib.check(L.sf_grad_jk(fb.handle, p[2], _ptr(apart), prec, 0.0, 0.0, _stream_ptr()))
    fb.set_profiling(profiling)
    _lib.check(L.sf_grad_rhf(fb.handle, p[0], p[1], 5, p[2], p[3], _ptr(both), prec, 0.0, 0.0, _stream_ptr()))
    assert (both - apart).abs().max() <= 1e-11 * apart.abs().max()
    with pytest.raises(Exception):   # the shells reference five nuclei
        _lib.check(L.sf_grad_rhf(fb.handle, p[0], p[1], 4, p[2], p[3], _ptr(both), prec, 0.0, 0.0, _stream_ptr()))
    fb.close()


CLASSES = [(a, b, c, d) for a in range(3) for b in range(a + 1) for c in range(3) for d in range(c + 1)
           if (a * (a + 1) // 2 + b) >= (c * (c + 1) // 2 + d)]


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("df", 1e-11), ("fp32", 3e-5)])
@pytest.mark.parametrize("cls", CLASSES, ids=lambda c: "%d%d%d%d" % c)
def test_fock_splits_by_class(cuda, cls, precision, tol):
    """J and K of four shells of one class against the oracle, for primitive splits from one lane group to
    more sub-groups than primitive quartets (digestion by one lane, all lanes of a quartet, whole CTAs).
    D has random signs, so an element's 400 terms add their errors up to 20 times one: 2^-44 (double-float) or
    less gives 2e-12 of the largest element, 3e-6 per FP32 integral 6e-5 of the largest term, a few of which
    make an element: 1e-11 and 3e-5."""
    from segfault_py_gb300.fock import FockBuilder
    table = _table(list(cls), [3, 2, 2, 3], 40 + sum(3 ** i * l for i, l in enumerate(cls)), 2.0)
    D = _sym(sum((l + 1) * (l + 2) // 2 for l in cls), 3)
    J, K = O.jk_direct(_cgfs(table), D)
    fb = FockBuilder(table, device=cuda, cutoff=0.0, precision=precision)
    Dd = torch.tensor(D, device=cuda)
    for split in (1, 2, 4, 8, 32, 128, 512):
        fb.set_tuning([dict(cls=c, precision=k, cost=n, split=split, ms_default=0.0, ms_tuned=0.0)
                       for c in range(21) for k in range(3) for n in range(1, 82)])
        for got, ref in zip(fb.jk(Dd), (J, K)):
            assert np.abs(got.cpu().numpy() - ref).max() <= tol * np.abs(ref).max(), split
    fb.close()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-6), ("df", 1e-6), ("fp32", 1e-4)])
@pytest.mark.parametrize("cls", CLASSES, ids=lambda c: "%d%d%d%d" % c)
def test_two_electron_gradient_by_class(cuda, cls, precision, tol):
    """All quartets of four shells of one class against central differences of the oracle's two-electron
    energy at a fixed density (no screening)."""
    from segfault_py_gb300 import _lib
    from segfault_py_gb300.fock import FockBuilder, _ptr, _stream_ptr
    table = _table(list(cls), [2, 1, 2, 1], sum(3 ** i * l for i, l in enumerate(cls)), 2.0)
    n = sum((l + 1) * (l + 2) // 2 for l in cls)
    D = _sym(n, 7)

    def energy(x):
        J, K = O.jk_direct(_cgfs(dict(table, center=x)), D)
        return 0.5 * np.sum(D * (J - 0.5 * K))

    fb = FockBuilder(table, device=cuda, cutoff=0.0)
    fb.set_density_screening(grad=False)
    Dd = torch.tensor(D, device=cuda)
    g = torch.zeros(12, dtype=torch.float64, device=cuda)
    _lib.check(_lib.lib().sf_grad_jk(fb.handle, _ptr(Dd), _ptr(g), _lib.PRECISION[precision], 0.0, 0.0, _stream_ptr()))
    g = g.cpu().numpy().reshape(4, 3)
    fb.close()
    assert np.abs(g.sum(axis=0)).max() <= tol * np.abs(g).max()
    x = table["center"]
    for a, k in [(0, 0), (1, 1), (2, 2), (3, 0)]:
        h = np.zeros_like(x)
        h[a, k] = 1e-4
        fd = (energy(x + h) - energy(x - h)) / 2e-4
        assert abs(fd - g[a, k]) <= tol * np.abs(g).max(), (a, k, fd, g[a, k])


@pytest.mark.parametrize("kmax", [1, 3, 4, 6])
@pytest.mark.parametrize("cls", [(0, 0, 0, 0), (1, 0, 1, 0), (1, 1, 1, 1), (2, 1, 2, 0), (2, 2, 2, 2)],
                         ids=lambda c: "%d%d%d%d" % c)
def test_raw_integral_splits(cuda, cls, kmax):
    """kmax^4 primitive quartets (1, 81, 256, 1296) from one to thousands per lane group: a lane or warp, a
    CTA and a cluster per quartet, in FP64, double-float and FP32, with the bounds of the random-shell test."""
    from segfault_py_gb300.fock import FockBuilder
    table = _table(list(cls) + list(cls), [kmax] * 8, 20 + kmax, 1.5, 0.3, 30.0)
    q = np.array([[0, 1, 2, 3], [4, 1, 6, 3], [0, 5, 2, 7]], dtype=np.int32)
    fb = FockBuilder(table, device=cuda)
    got = {p: fb.eri_quartets(q, precision=p) for p in ("fp64", "df", "fp32")}
    fb.close()
    O.use_exact_roots(True)
    try:
        for k, row in enumerate(q):
            cg = [_shell_cgfs(table, s) for s in row]
            n = np.cumsum([0] + [len(c) for c in cg])
            idx = [[n[0] + i, n[1] + j, n[2] + m, n[3] + l] for i in range(len(cg[0])) for j in range(len(cg[1]))
                   for m in range(len(cg[2])) for l in range(len(cg[3]))]
            ref = O.eri_list(sum(cg, []), np.array(idx)).reshape(got["fp64"][k].shape)
            for p, tol in (("fp64", 1e-10), ("df", 1e-10), ("fp32", 1e-4)):
                assert np.abs(got[p][k] - ref).max() <= tol * np.abs(ref).max(), (p, k)
    finally:
        O.use_exact_roots(False)


@pytest.mark.parametrize("distance", [0.0, 4.0, 12.0, 60.0])
def test_dropped_primitive_pairs(cuda, distance):
    """Contractions of tight and diffuse functions at a distance where none, some or all but one primitive
    pair (at 60 bohr every product underflows) are negligible: integrals as from the full contraction."""
    from segfault_py_gb300.fock import FockBuilder
    table = _table([0, 2, 1, 0], [4, 4, 4, 4], 9, 0.5)
    table["exps"] = np.tile(np.array([4000.0, 300.0, 12.0, 0.4]), 4)
    table["center"][[1, 3], 0] += distance
    q = np.array([[0, 1, 2, 3], [0, 0, 1, 3], [0, 2, 1, 3], [2, 1, 2, 1]], dtype=np.int32)
    fb = FockBuilder(table, device=cuda)
    blocks = {p: fb.eri_quartets(q, precision=p) for p in ("fp64", "df")}
    fb.close()
    O.use_exact_roots(True)
    try:
        for k, row in enumerate(q):
            cg = [_shell_cgfs(table, s) for s in row]
            n = np.cumsum([0] + [len(c) for c in cg])
            idx = [[n[0] + i, n[1] + j, n[2] + m, n[3] + l] for i in range(len(cg[0])) for j in range(len(cg[1]))
                   for m in range(len(cg[2])) for l in range(len(cg[3]))]
            ref = O.eri_list(sum(cg, []), np.array(idx)).reshape(blocks["fp64"][k].shape)
            for p in ("fp64", "df"):
                assert np.all(np.isfinite(blocks[p][k]))
                assert np.abs(blocks[p][k] - ref).max() <= 1e-10 * np.abs(ref).max() + 1e-30, (p, k)
    finally:
        O.use_exact_roots(False)
