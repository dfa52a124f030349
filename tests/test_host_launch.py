"""What the library launches, copies and waits for, on a recording stand-in for the CUDA runtime."""
import pytest

import fake_cuda
from segfault_py_gb300 import geometry as G
from segfault_py_gb300.molecule import Molecule


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_cuda.make(str(tmp_path_factory.mktemp("fake")))


def _table(n=2, basis="6-31g*"):
    return Molecule.from_geometry(*G.water_cluster(n, seed=1), basis).shell_table()


def test_lists_of_a_failed_build_are_not_kept(fake):
    """Lists that could not be cut completely (no memory) are cut again by the next call, whatever its mode."""
    h = fake.handle(_table())
    fake.ok(fake.fock(h, "fp64"))
    good = [(r.cls, r.kind, r.n, r.split) for r in fake.launches()]
    assert good
    failed = 0
    for k in range(40):   # every allocation of the other mode's lists in turn
        fake.L.fake_fail_malloc(k)
        rc = fake.fock(h, "mixed", cut=0.0)
        fake.L.fake_fail_malloc(-1)
        fake.log()
        if rc == 0:
            break
        failed += 1
        assert fake.L.sf_slice_count(h) == 0
        fake.ok(fake.fock(h, "fp64"))
        assert [(r.cls, r.kind, r.n, r.split) for r in fake.launches()] == good
    assert failed > 0
    fake.L.sf_destroy(h)


@pytest.mark.parametrize("profiling", [0, 1, 2])
@pytest.mark.parametrize("then", ["precision", "cutoff", "partition", "tuning", "schwarz", "forces"])
def test_lists_in_use_are_not_overwritten(fake, then, profiling):
    """Calls return before their kernels end: lists (and pair tables) that launched kernels read are overwritten
    only after a wait for the streams those run on.  The copies do not order themselves behind such streams."""
    h = fake.handle(_table())
    fake.ok(fake.L.sf_set_profiling(h, profiling))
    fake.ok(fake.fock(h, "fp64"))
    first = fake.log()
    assert not [r for r in first if r.what == fake_cuda.SYNC]   # nothing to wait for
    last = {r.stream: i for i, r in enumerate(first) if r.what == fake_cuda.LAUNCH}   # of each stream
    fake.ok(fake.fock(h, "fp64"))   # the same lists: no copy, no wait
    assert not [r for r in fake.log() if r.what in (fake_cuda.SYNC, fake_cuda.MEMCPY)]
    if then == "partition":
        fake.ok(fake.L.sf_set_partition(h, 0, 2))
    if then == "tuning":
        fake.ok(fake.L.sf_set_tuning(h, None, 0))
    if then == "schwarz":
        fake.ok(fake.L.sf_schwarz(h, None, 0x55))
    elif then == "forces":
        fake.ok(fake.forces(h, "df"))
    else:
        fake.ok(fake.fock(h, "df" if then == "precision" else "fp64", cut=1e-9 if then == "cutoff" else 1e-12))
    log = fake.log()
    copy = min(i for i, r in enumerate(log) if r.what == fake_cuda.MEMCPY and (then != "schwarz" or r.stream == 0))
    waited = {r.stream for r in log[:copy] if r.what == fake_cuda.SYNC}
    for i, r in enumerate(first):   # a stream waited for may itself have waited for another one's event
        if r.what == fake_cuda.WAIT and r.stream in waited:
            waited |= {e.stream for j, e in enumerate(first[:i]) if e.what == fake_cuda.RECORD and e.list == r.list
                       and j > last.get(e.stream, -1)}
    assert set(last) <= waited
    fake.L.sf_destroy(h)


def _kinds(fake, table, scale=1.0, cut=1e-12):
    h = fake.handle(table, q_scale=scale)
    fake.ok(fake.fock(h, "fp64", cut=cut * scale * scale))
    n = {}
    for r in fake.launches():
        n[r.cls, r.kind] = n.get((r.cls, r.kind), 0) + r.n
    fake.L.sf_destroy(h)
    return n


def test_double_float_part_follows_the_largest_bound(fake):
    """The FP64 mode's double-float part is what is small against the molecule's own largest quartets: scaling every
    function moves no quartet, and bounds or primitives outside FP32's range leave everything in FP64."""
    table = _table(6)
    ref = _kinds(fake, table)
    assert {k for _, k in ref} == {0, 2}
    for s in (2.0 ** -10, 2.0 ** -3, 2.0 ** 4):
        assert _kinds(fake, table, s) == ref
    for s in (2.0 ** -40, 2.0 ** 40):
        assert {k for _, k in _kinds(fake, table, s)} == {0}
    for key, v in (("exps", 1e30), ("exps", 1e-30), ("coefs", 1e25)):
        t = dict(table, **{key: table[key].copy()})
        t[key][3] = v
        assert {k for _, k in _kinds(fake, t)} == {0}, key
    # no quartet of 2e-4 of the largest bound (1 here) or more is in it
    assert {k for _, k in _kinds(fake, table, cut=2e-4)} == {0}


@pytest.mark.parametrize("precision,waters", [("mixed", 3), ("mixed_df", 3), ("mixed_df", 8)])
def test_demoted_launches_share_the_streams(fake, precision, waters):
    """The FP32 launches of demoted quartets are spread over the FP32 streams, by estimated cost: more of them than
    streams, they use at least half of the streams."""
    h = fake.handle(_table(waters))
    fake.ok(fake.forces(h, precision, cut32=1e-2))
    runs = {}
    for r in fake.launches():
        runs.setdefault((r.stream, r.cls, r.kind, r.count % 32), 0)   # the counts of a slice: kept, demoted, ...
    base = min(c for _, _, k, c in runs if k != 1)
    demoted = [s for s, _, k, c in runs if k == 1 and c == (base + 8) % 32]
    low = {s for s, _, k, _ in runs if k == 1}
    assert len(demoted) > len(low) > 1
    assert 2 * len(set(demoted)) >= len(low)
    fake.L.sf_destroy(h)


def test_gradient_launches_of_the_double_float_part(fake):
    """Gradients keep in double-float only what the classification leaves there: every such launch has an FP64 one
    of what it takes out, and with the classification off or an FP32 tier beside it the whole part is FP64."""
    h = fake.handle(_table(6))
    fake.ok(fake.fock(h, "fp64"))
    assert {r.kind for r in fake.launches()} == {0, 2}
    fake.ok(fake.forces(h, "fp64"))
    runs = fake.launches()
    dd = {(r.cls, r.count + 8) for r in runs if r.kind == 2}   # the counts of a slice: kept, taken out, ...
    assert dd and dd <= {(r.cls, r.count) for r in runs if r.kind == 0}
    fake.ok(fake.L.sf_set_density_screening(h, 0, -1.0, -1.0, -1.0))
    fake.ok(fake.forces(h, "fp64"))
    assert {r.kind for r in fake.launches()} == {0}
    fake.ok(fake.L.sf_set_density_screening(h, 2, -1.0, -1.0, -1.0))
    fake.ok(fake.forces(h, "mixed"))
    assert {r.kind for r in fake.launches()} == {0, 1}
    fake.L.sf_destroy(h)


@pytest.mark.parametrize("waters,part", [(2, False), (6, True)])
def test_measured_times_order_the_launches(fake, waters, part):
    """Measured launch times decide the order and the streams, also where part of the build is in double-float,
    which is not tuned and goes by its estimate."""
    from segfault_py_gb300 import _lib
    h = fake.handle(_table(waters))
    costs = range(1, 36 * 36 + 1)
    entries = [_lib.TuneEntry(cls=c, precision=0, cost=k, split=1, ms_default=1.0, ms_tuned=1e4 if c == 20 else 1.0)
               for c in range(21) for k in costs]
    arr = (_lib.TuneEntry * len(entries))(*entries)
    fake.ok(fake.L.sf_set_tuning(h, arr, len(entries)))
    fake.ok(fake.fock(h, "fp64"))
    runs = fake.launches()
    assert any(r.kind == 2 for r in runs) == part
    assert [r.cls for r in runs if r.kind == 0][0] == 20   # (dd|dd), the cheapest by its estimate
    if part:   # estimates in the measured times' unit: neither all before nor all after the timed launches
        kinds = [r.kind for r in runs]
        assert kinds != sorted(kinds) and kinds != sorted(kinds, reverse=True)
    fake.L.sf_destroy(h)


@pytest.mark.parametrize("precision", ["fp64", "mixed_df"])
@pytest.mark.parametrize("fill", [0, 1, 16])
def test_gradient_splits_do_not_follow_the_tuned_fill(fake, precision, fill):
    """The fill target that the autotuner finds for a mode's Fock builds (0: no extra split) is not the gradient's:
    its splits go by the work per lane of the whole GPU."""
    from segfault_py_gb300 import _lib
    h = fake.handle(_table(3))

    def loads():
        fake.ok(fake.forces(h, precision, cut32=1e-2))
        out = {}
        for r in fake.launches():
            out.setdefault((r.cls, r.kind), set()).add(r.rel_load)
        return out

    ref = loads()
    arr = (_lib.TuneEntry * 2)(*[_lib.TuneEntry(cls=c, precision=_lib.PRECISION[precision], cost=0, split=fill)
                                 for c in (-1, -2)])
    fake.ok(fake.L.sf_set_tuning(h, arr, 2))
    assert loads() == ref
    fake.L.sf_destroy(h)


NO_THREADS = r"""
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
int refuse_threads = 0;
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
  static int (*real)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
  if (refuse_threads) return EAGAIN;
  if (!real) real = (int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create");
  return real(t, a, f, arg);
}
"""

NO_THREADS_RUN = """
import ctypes, sys
sys.path[:0] = [%(tests)r, %(repo)r]
import fake_cuda
from test_host_launch import _table
fake = fake_cuda.Fake(%(lib)r)
ctypes.c_int.in_dll(ctypes.CDLL(%(pre)r), "refuse_threads").value = 1
h = fake.handle(_table(6))
fake.ok(fake.fock(h, "fp64"))
print(len(fake.launches()))
"""


def test_no_threads_to_be_had(fake, tmp_path):
    """Where the system gives no more threads, the tables and the quartet lists are made on the caller's."""
    import os
    import subprocess
    import sys
    src, pre = tmp_path / "nothreads.c", tmp_path / "nothreads.so"
    src.write_text(NO_THREADS)
    subprocess.run(["gcc", "-D_GNU_SOURCE", "-shared", "-fPIC", str(src), "-o", str(pre), "-ldl"], check=True)
    here = os.path.dirname(os.path.abspath(__file__))
    code = NO_THREADS_RUN % dict(tests=here, repo=os.path.dirname(here), lib=fake.path, pre=str(pre))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=str(pre)))
    assert r.returncode == 0, r.stderr
    h = fake.handle(_table(6))
    fake.ok(fake.fock(h, "fp64"))
    assert int(r.stdout) == len(fake.launches()) > 0
    fake.L.sf_destroy(h)
