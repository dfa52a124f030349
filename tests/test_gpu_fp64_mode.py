"""What the FP64 mode runs in double-float."""
import numpy as np
import pytest
import torch

from test_gpu_kernel_edges import _sym

pytestmark = pytest.mark.gpu

CUT, TAIL = 1e-9, 2e-4


@pytest.fixture(scope="module")
def water(cuda):
    from segfault_py_gb300 import geometry as G
    from segfault_py_gb300.fock import FockBuilder
    from segfault_py_gb300.molecule import Molecule
    mol = Molecule.from_geometry(*G.water_cluster(5, seed=4), "6-31g*")
    fb = FockBuilder(mol, device=cuda, cutoff=CUT, precision="fp64")
    fb.set_density_screening(grad=True, grad_drop_cutoff=0.0)
    yield fb, torch.tensor(_sym(mol.nao, 5), device=cuda)
    fb.close()


def _forces(fb, D):
    """The two-electron forces and (class, kind) -> quartets of the launches."""
    from segfault_py_gb300 import _lib
    from segfault_py_gb300.fock import _ptr, _stream_ptr
    g = torch.zeros(3 * fb.mol.natom, dtype=torch.float64, device=D.device)
    _lib.check(_lib.lib().sf_grad_jk(fb.handle, _ptr(D), _ptr(g), _lib.PRECISION["fp64"], CUT, 0.0, _stream_ptr()))
    n = {}
    for s in fb.slice_info():
        n[s["cls"], s["precision"]] = n.get((s["cls"], s["precision"]), 0) + s["quartets"]
    return g, n


def test_gradient_part_by_derivative_bound(water):
    """A quartet's gradient stays in double-float while its density-weighted bound, times the square roots of its
    largest exponents, is below the threshold: counted here from the Schwarz bounds."""
    fb, D = water
    fb.jk(D)
    part = {s["cls"] for s in fb.slice_info() if s["precision"] == 2}
    assert part
    _, n = _forces(fb, D)
    t, l = fb.table, fb.l
    off = np.append(fb.ao_offset, fb.nao)
    M = D.abs().cpu().numpy()
    M = np.array([[M[off[a]:off[a + 1], off[b]:off[b + 1]].max() for b in range(fb.nshell)] for a in range(fb.nshell)])
    s = np.sqrt([t["exps"][o:o + k].max() for o, k in zip(t["prim_offset"], t["nprim"])])
    pairs = [np.array([(a, b) for a in range(fb.nshell) for b in range(fb.nshell)
                       if (l[a], l[b]) == x and (l[a] > l[b] or a >= b)]) for x in
             [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2)]]
    top = fb.q.max() ** 2
    for cls in part:
        x = next(k for k in range(6) if k * (k + 1) // 2 <= cls < (k + 1) * (k + 2) // 2)
        y = cls - x * (x + 1) // 2
        A, B = pairs[x], pairs[y]
        q = fb.q[A[:, 0], A[:, 1]][:, None] * fb.q[B[:, 0], B[:, 1]]
        a, b, c, d = A[:, :1], A[:, 1:], B[:, 0], B[:, 1]
        bound = q * (0.5 * M[a, b] * M[c, d] + 0.125 * (M[a, c] * M[b, d] + M[a, d] * M[b, c]))
        low = (q >= CUT) & (q < TAIL * top) & (bound * (s[a] + s[b] + s[c] + s[d]) < TAIL * top * M.max() ** 2)
        if x == y:   # unordered pairs of pairs: the matrix is symmetric
            count = (low.sum() + np.diag(low).sum()) / 2
        else:
            count = low.sum()
        assert abs(n[cls, 2] - count) <= 1e-4 * count + 2, cls   # FP32 rounding of the bounds at the threshold


def test_gradient_part_follows_the_density(water):
    """The threshold scales with the density; a density near the ends of FP32's range, or not a number, leaves
    everything in FP64 and the forces are what FP64 makes of it."""
    fb, D = water
    g, n = _forces(fb, D)
    assert any(k == 2 for _, k in n)
    for e in (-20, 20):
        g2, n2 = _forces(fb, D * 2.0 ** e)
        assert n2 == n
        # equal quartets and roundings, FP64 sums of fewer than 1e5 terms in another order
        assert float((g2 * 2.0 ** (-2 * e) - g).abs().max()) <= 1e-11 * float(g.abs().max())
    for e in (-40, 40):
        g2, n2 = _forces(fb, D * 2.0 ** e)
        assert not any(v for (_, k), v in n2.items() if k == 2)
        # against the double-float part's 2^-44: fewer than 1e5 terms
        assert float((g2 * 2.0 ** (-2 * e) - g).abs().max()) <= 1e-10 * float(g.abs().max())
    bad = D.clone()
    bad[3, 4] = bad[4, 3] = float("nan")
    g2, n2 = _forces(fb, bad)
    assert not any(v for (_, k), v in n2.items() if k == 2) and torch.isnan(g2).any()


@pytest.mark.parametrize("call", ["handle", "noalloc"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_density_outside_the_range_of_fp32(water, precision, call):
    """J and K are linear in the density over FP64's whole range, with part of the build in double-float: powers of
    two change no digits, FP64 sums of fewer than 1e4 terms come in another order.  Not a number, or infinite, in one
    element: so are J and K.  The output may be the density's own matrix."""
    from segfault_py_gb300 import _lib
    from segfault_py_gb300.fock import _ptr, _stream_ptr
    fb, D = water
    n, cut32 = fb.nao, 1e-6

    def jk(D, J=None, K=None):
        J, K = (torch.full_like(D, 7.0) if m is None else m for m in (J, K))
        run = _lib.lib().sf_fock_jk_noalloc if call == "noalloc" else \
            lambda *a: _lib.lib().sf_fock_jk(*a[:-1], None, a[-1])
        _lib.check(run(fb.handle, _ptr(D), _ptr(J), _ptr(K), _lib.PRECISION[precision], CUT, cut32, _stream_ptr()))
        return J, K

    ref = fb.jk(D, precision=precision, fp32_cutoff=cut32)
    assert any(s["precision"] == 2 and s["quartets"] for s in fb.slice_info())
    for e in (0, -30, 30, -140, 140, -900, 900):
        for got, r in zip(jk(D * 2.0 ** e), ref):
            got = got * 2.0 ** (-e // 2) * 2.0 ** (-e - -e // 2)
            assert float((got - r).abs().max()) <= 1e-12 * float(r.abs().max()), e
    for bad in (float("nan"), float("inf")):
        B = D.clone()
        B[2, 9] = B[9, 2] = bad
        assert not any(torch.isfinite(m).any() for m in jk(B))
    own = D.clone()
    for got, r in zip(jk(own, J=own), ref):
        assert float((got - r).abs().max()) <= 1e-12 * float(r.abs().max())
    both = D.clone()
    jk(D, J=both, K=both)   # one matrix for both: K
    assert float((both - ref[1]).abs().max()) <= 1e-12 * float(ref[1].abs().max())
    assert torch.isfinite(jk(torch.zeros_like(D))[0]).all()


def test_double_float_part_by_class(cuda):
    """All 21 classes with a double-float part against the same quartets in FP64 throughout (a shell outside FP32's
    range, uncoupled, keeps that handle there).  The part's terms carry 2^-44 and add up to at most ten times the
    largest element: 1e-12 of it in J and K, 1e-11 in the forces, whose terms reach further above their sums."""
    from segfault_py_gb300 import _lib
    from segfault_py_gb300.fock import FockBuilder, _ptr, _stream_ptr
    from test_gpu_kernel_edges import _table
    ls = [0, 1, 2] * 36
    table = _table(ls, [2, 1, 1] * 36, 6, 9.0)
    n, m = sum((l + 1) * (l + 2) // 2 for l in ls), len(ls)
    more = dict(table, l=np.append(table["l"], 0), nprim=np.append(table["nprim"], 1), atom=np.append(table["atom"], m),
                ao_offset=np.append(table["ao_offset"], n), center=np.vstack([table["center"], [[4.0, 4.0, 4.0]]]),
                prim_offset=np.append(table["prim_offset"], table["prim_offset"][-1] + 1),
                exps=np.append(table["exps"], 1e10), coefs=np.append(table["coefs"], 1e-3))
    more = {k: v.astype(table[k].dtype) for k, v in more.items()}
    D = np.zeros((n + 1, n + 1))
    D[:n, :n] = _sym(n, 9)
    out = []
    for t, size in ((table, n), (more, n + 1)):
        fb = FockBuilder(t, device=cuda, cutoff=1e-12, precision="fp64")
        Dd = torch.tensor(np.ascontiguousarray(D[:size, :size]), device=cuda)
        J, K = fb.jk(Dd)
        part = {s["cls"] for s in fb.slice_info() if s["precision"] == 2}
        assert part == (set(range(21)) if size == n else set())
        g = torch.zeros(3 * (m + 1), dtype=torch.float64, device=cuda)
        _lib.check(_lib.lib().sf_grad_jk(fb.handle, _ptr(Dd), _ptr(g), _lib.PRECISION["fp64"], 1e-12, 0.0,
                                         _stream_ptr()))
        out.append((J[:n, :n].clone(), K[:n, :n].clone(), g[:3 * m].clone()))
        fb.close()
    for a, b, tol in zip(*out, (1e-12, 1e-12, 1e-11)):
        assert float((a - b).abs().max()) <= tol * float(b.abs().max())
