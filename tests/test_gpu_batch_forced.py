"""The batched engine's switch for the values per thread of a run-time length, on a GPU.

BWPM_RT_E takes the kernel with that E wherever it can run the length, the general forms (16, 20, 24
and 30) among them at lengths that also have a plan with equal outer radices. The class's threads
tell which kernel was taken; results are held to the numpy oracle at the complex64 contract
(relative L2 ≤ 1e-4).
"""

from __future__ import annotations

import pytest

from conftest import rel_l2
from test_gpu_solver_sharing import _line

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,e", [(1600, 4), (1600, 5), (900, 6), (1600, 8), (810, 9), (1600, 10), (1440, 12),
                                  (900, 15), (1600, 16), (1600, 20), (1152, 24), (900, 30), (2400, 30)])
def test_forced_values_per_thread(monkeypatch, ny, e):
    from bwpm_b200.batch import Batch2D
    from oracle import port

    (_, _, dy, dx, dz, k0, idx, labels, before, mask), field = _line(ny, 12, True)
    monkeypatch.setenv("BWPM_RT_E", str(e))
    b = Batch2D(0)
    b.add(ny, dy, dz, k0, idx, labels, before, mask, field, 1)
    b.prepare()
    (c,) = b.classes()
    assert c["threads"] == (ny // e + 31) // 32 * 32
    b.run()
    got = b.result(0)
    ref = port.Solver(ny, 1, dy, dx, dz, k0, idx, labels, before, mask).run(field, 1)
    for key in ("transmitted", "reflected"):
        assert rel_l2(got[key], ref[key][:, 0]) < 1e-4, key
