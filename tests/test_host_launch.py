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
