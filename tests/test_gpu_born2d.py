"""The 2D Born slab kernel (bwpm_b200/csrc/born2d.cuh) on a GPU.

A slab's GMRES, its increment, the step itself and the back-scatter run in one launch, the line
split over 1, 2, 4 or 8 CTAs with compiled and run-time lengths per CTA. A volume with δn in slabs
of two hosts (one absorbing), slabs without δn, a tilted interface (steps of several passes that the
launch does not take over) and a mask, both components, is held to the numpy oracle and to the
multi-kernel form (BWPM_GMRES=graph): FP64 at the drop-in contract (1e-10), complex64 at its own
(relative L2 ≤ 1e-4).
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = {64: 1e-10, 32: 1e-4}


def _case(ny: int, masked: bool):
    rng = np.random.default_rng(ny)
    lam = 0.633e-3
    nz, dy, dz = 9, lam / 8, lam / 10
    y = (np.arange(ny) - ny // 2) * dy
    labels = np.zeros((nz, ny), np.int32)
    labels[4, ny // 3:] = 1  # an interface across the line inside slab 4
    labels[5:] = 1
    fl = np.zeros((nz, ny), complex)
    fl[1:4] = 0.01 * rng.standard_normal((3, ny))
    fl[4, : ny // 3 - 2] = 0.01 * rng.standard_normal(ny // 3 - 2)
    fl[6:8] = 0.01 * rng.standard_normal((2, ny))
    field = np.zeros((ny, 1, 2), complex)
    beam = np.exp(-((y / (ny * dy / 5)) ** 2) + 0.3j * y / dy)
    field[:, 0, 0] = beam
    field[:, 0, 1] = 0.4j * beam * rng.uniform(0.9, 1.1, ny)
    mask = np.exp(-((y / (0.45 * ny * dy)) ** 8))[:, None] if masked else None
    args = (ny, 1, dy, 1.0, dz, 2 * np.pi / lam, np.array([1.5, 1.4 + 0.02j]), labels[:, :, None],
            1.0 + 0j, mask)
    return args, field, fl[:, :, None]


@pytest.mark.parametrize("ny,masked", [(64, True), (144, False), (250, True), (512, False),
                                       (640, True), (1000, False), (1024, True), (1536, False),
                                       (2048, True), (2430, False), (3072, True), (3584, False),
                                       (4096, True), (6144, False)])
def test_born_slab_matches_graph_and_oracle(monkeypatch, ny, masked):
    from bwpm_b200 import _core
    from oracle import port

    args, field, fl = _case(ny, masked)
    for iters, keep in ((0, [0, 3, 9]), (2, [0, 2, 5, 9])):
        ref = port.Solver(*args, fluctuation=fl).run(field, iters, keep)
        for prec in (64, 32):
            for mode in (None, "graph"):
                if mode:
                    monkeypatch.setenv("BWPM_GMRES", mode)
                else:
                    monkeypatch.delenv("BWPM_GMRES", raising=False)
                s = _core.CudaSolver(*args, 0, fluctuation=fl, precision=prec)
                got = s.run(field, iters, keep)
                tol = TOL[prec]
                assert rel_l2(got["transmitted"], ref["transmitted"]) < tol, (prec, mode)
                for q in keep:
                    assert rel_l2(got["forward"][q], ref["forward"][q]) < tol, (prec, mode, q)
                if iters:
                    assert rel_l2(got["reflected"], ref["reflected"]) < tol, (prec, mode)
                    for q in keep:
                        if np.linalg.norm(ref["backward"][q]) > 0:
                            assert rel_l2(got["backward"][q], ref["backward"][q]) < tol, (prec, mode, q)
                again = s.run(field, iters, [])
                assert np.array_equal(again["transmitted"], got["transmitted"])
                assert s.stats()["gmres_applies"] > 0


def test_born_slab_restart_limit_raises(monkeypatch):
    """A tolerance of 0 ends after 100 restarts with RuntimeError (cpp/src/solver.cpp:341-342); the
    next solver on the device runs normally."""
    from bwpm_b200 import _core

    monkeypatch.delenv("BWPM_GMRES", raising=False)
    ny, lam = 1024, 0.633e-3
    dy, dz = lam / 8, lam / 10
    y = (np.arange(ny) - ny // 2) * dy
    field = np.zeros((ny, 1, 2), complex)
    field[:, 0, 0] = np.exp(-((y / (64 * dy)) ** 2))
    labels = np.zeros((1, ny, 1), np.int32)
    fl = 0.01 * np.random.default_rng(3).standard_normal((1, ny, 1)) + 0j
    args = (ny, 1, dy, 1.0, dz, 2 * np.pi / lam, np.array([1.5 + 0j]), labels, 1.0 + 0j, None)
    with pytest.raises(RuntimeError, match="GMRES did not converge"):
        _core.CudaSolver(*args, 0, fluctuation=fl, gmres_tol=0.0).run(field, 0, [])
    r = _core.CudaSolver(*args, 0, fluctuation=fl).run(field, 0, [])
    assert np.all(np.isfinite(r["transmitted"])) and np.linalg.norm(r["transmitted"]) > 0
