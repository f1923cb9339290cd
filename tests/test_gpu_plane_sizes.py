"""The register-resident 3D step kernels (bwpm_b200/csrc/plane_rf.cuh) over lateral sizes, on a GPU.

Compiled lengths mixed with run-time ones (n = E²·m), odd and even, square and not, with one and
two lines per CTA, down to the smallest: a volume of three materials (one absorbing) with a
tilted, curved front (steps of several passes, rows in which a pass's pair does not occur), a
planar back face, a mask and both components, two iterations. FP64 is held to the general kernels
(BWPM_3D_KERNELS=general) and, for small planes, to the numpy oracle at the drop-in contract
(1e-10); complex64 to FP64 at its contract (relative L2 ≤ 1e-4).
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _case(ny: int, nx: int, nz: int):
    lam = 0.633e-3
    d, dz = lam / 6, lam / 8
    y = (np.arange(ny) - ny // 2) * d
    x = (np.arange(nx) - nx // 2) * d
    front = 3 + np.floor(3 * (np.arange(ny)[:, None] / ny) * np.ones((1, nx))
                         + 1.5 * np.cos(np.pi * x / (nx * d))[None, :]).astype(int)
    labels = np.zeros((nz, ny, nx), np.int32)
    for j in range(nz):
        labels[j][j >= front] = 1
    labels[nz - 2:] = 2
    r2 = (y[:, None] / (ny * d / 4)) ** 2 + (x[None, :] / (nx * d / 4)) ** 2
    field = np.zeros((ny, nx, 2), complex)
    field[..., 0] = np.exp(-r2 + 0.2j * y[:, None] / d)
    field[..., 1] = 0.5j * np.exp(-r2 - 0.1j * x[None, :] / d)
    mask = np.exp(-r2 / 16)
    args = (ny, nx, d, d, dz, 2 * np.pi / lam, np.array([1.0, 1.5, 1.2 + 0.05j]), labels,
            1.0 + 0j, mask)
    return args, field


@pytest.mark.parametrize("ny,nx", [(4, 8), (9, 4), (16, 36), (49, 50), (45, 36), (64, 256),
                                   (243, 125), (375, 250), (256, 384), (384, 100), (768, 18),
                                   (18, 1024), (1600, 16), (16, 2187), (300, 512), (98, 27)])
def test_sizes_match_general_kernels_and_oracle(monkeypatch, ny, nx):
    from bwpm_b200 import _core
    from oracle import port

    nz, iters, keep = 10, 2, [0, 4, 10]
    args, field = _case(ny, nx, nz)
    got = {}
    for name, prec in (("rf", 64), ("general", 64), ("rf", 32)):
        if name == "general":
            monkeypatch.setenv("BWPM_3D_KERNELS", "general")
        else:
            monkeypatch.delenv("BWPM_3D_KERNELS", raising=False)
        got[name, prec] = _core.CudaSolver(*args, 0, precision=prec).run(field, iters, keep)
    refs = [got["general", 64]]
    if ny * nx <= 16384:
        refs.append(port.Solver(*args).run(field, iters, keep))
    for ref in refs:
        for prec, tol in ((64, 1e-10), (32, 1e-4)):
            r = got["rf", prec]
            for key in ("transmitted", "reflected"):
                assert rel_l2(r[key], ref[key]) < tol, (prec, key)
            for q in keep:
                assert rel_l2(r["forward"][q], ref["forward"][q]) < tol, (prec, q)
            assert rel_l2(r["backward"][4], ref["backward"][4]) < tol, prec
    r = got["rf", 64]
    assert np.array_equal(r["transmitted_iter"][-1], r["transmitted"])
    assert np.array_equal(r["reflected_iter"][-1], r["reflected"])
    for it in range(iters):  # the earlier sweep's planes, downloaded while later sweeps run
        for key in ("transmitted_iter", "reflected_iter"):
            assert rel_l2(r[key][it], got["general", 64][key][it]) < 1e-10, (key, it)
