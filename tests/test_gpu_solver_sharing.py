"""Solvers that are alive together and share kernel functions, on a GPU.

One kernel function serves many sizes (run-time lengths of one E, a compiled length with and
without a mask), each with its own dynamic shared memory, and the limit of that memory belongs to
the function on the device, not to the solver. So solvers made from the largest size to the
smallest must all still run afterwards, with the bits of a run right after their own set-up.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAM = 0.633e-3
K0 = 2 * np.pi / LAM


def _line(ny: int, nz: int, masked: bool):
    y = (np.arange(ny) - ny // 2) * LAM / 8
    labels = np.zeros((nz, ny, 1), np.int32)
    labels[nz // 3:, ny // 3:] = 1
    labels[nz // 2:] = 1
    field = np.zeros((ny, 1, 2), complex)
    field[:, 0, 0] = np.exp(-((y / (ny * LAM / 40)) ** 2))
    mask = np.exp(-((y / (ny * LAM / 18)) ** 8))[:, None] if masked else None
    return (ny, 1, LAM / 8, 1.0, LAM / 10, K0, np.array([1.0, 1.5 + 0j]), labels, 1.0 + 0j, mask), field


def _plane(ny: int, nx: int, nz: int):
    args, line = _line(ny, nz, True)
    labels = np.broadcast_to(args[7], (nz, ny, nx)).copy()
    field = np.broadcast_to(line, (ny, nx, 2)) * np.exp(-(np.linspace(-2, 2, nx) ** 2))[None, :, None]
    mask = np.broadcast_to(args[9], (ny, nx)).copy()
    return (ny, nx, LAM / 6, LAM / 6, LAM / 8, K0, args[6], labels, 1.0 + 0j, mask), field


def _case(kind: str, size):
    """(solver arguments, field, keyword arguments)"""
    if kind == "chain":
        return (*_line(size[0], 8, size[1]), {})
    if kind == "plane":
        return (*_plane(*size, 5), {})
    args, field = _line(size, 4, False)
    dn = 0.01 * np.random.default_rng(size).standard_normal((4, size, 1)) + 0j
    return args, field, {"fluctuation": np.where(args[7] == 0, dn, 0)}


SIZES = {
    "chain": [(n, m) for n in (8192, 6144, 4096, 3072, 2048, 1536, 1024, 768, 512, 384, 256)
              for m in (True, False)]
    + [(n, True) for n in (4050, 3645, 3600, 2430, 2400, 2187, 1944, 1620, 1600, 1215, 1080, 900, 800,
                           750, 600, 500, 400, 300, 225, 150, 100, 64, 36)],
    "born": [3584, 3200, 3000, 2800, 2560, 2430, 2048, 2000, 1920, 1500, 1280, 1000, 900, 640, 500, 400, 250],
    "plane": [(600, 375), (500, 500), (375, 250), (300, 320), (250, 150), (225, 225), (200, 192),
              (150, 100), (128, 64), (100, 75), (50, 25), (18, 36)],
}


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("kind", ["chain", "born", "plane"])
def test_solvers_alive_together(kind, precision):
    from bwpm_b200 import _core

    made = []
    for size in SIZES[kind]:
        args, field, kw = _case(kind, size)
        s = _core.CudaSolver(*args, 0, precision=precision, **kw)
        made.append((size, s, field, s.run(field, 1, [])))
    for size, s, field, first in made + made[::-1]:  # after the smallest was made, in both orders
        again = s.run(field, 1, [])
        for key in ("transmitted", "reflected"):
            assert np.array_equal(again[key], first[key]), (size, key)
