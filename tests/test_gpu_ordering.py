"""Calls in a row on a non-blocking stream, nothing waited for between them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_modes_back_to_back_on_a_stream(cuda):
    """Each mode's call re-cuts the quartet lists while the call before it may still run.  J and K as from calls
    that were waited for: sums of fewer than 1e4 terms in another order, 1e-12 of the largest element."""
    from segfault_py_gb300 import geometry as G
    from segfault_py_gb300.fock import FockBuilder
    from segfault_py_gb300.molecule import Molecule
    mol = Molecule.from_geometry(*G.water_cluster(6, seed=2), "6-31g*")
    A = np.random.default_rng(1).standard_normal((mol.nao, mol.nao))
    D = torch.tensor(0.1 * (A + A.T), device=cuda)
    modes = [("fp64", 0.0), ("df", 0.0), ("mixed_df", 1e-3), ("fp64", 1e-12), ("mixed", 1e-4), ("fp32", 0.0)]
    fb = FockBuilder(mol, device=cuda, cutoff=1e-11)
    ref = []
    for precision, c32 in modes:
        ref.append(fb.jk(D, precision=precision, fp32_cutoff=c32))
        torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        got = [fb.jk(D, precision=precision, fp32_cutoff=c32) for precision, c32 in modes * 2]
    stream.synchronize()
    for k, pair in enumerate(got):
        for a, b in zip(pair, ref[k % len(modes)]):
            assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max()), modes[k % len(modes)]
    fb.close()
