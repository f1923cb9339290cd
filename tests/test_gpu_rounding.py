"""Rounding error of the register-resident kernels against the kernels they replace, on a GPU.

Both compute the same transforms with other radices, so at one size and one input either can be
nearer to the exact result; over sizes and inputs these kernels must not be the further ones. Errors
against a more exact solution (complex64: the FP64 solver; FP64: a homogeneous medium in long double)
are compared pair by pair: the geometric mean of their ratio may exceed 1 by two of its standard
errors at most.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

LAM = 0.633e-3
K0 = 2 * np.pi / LAM


def _volume(ny: int, nx: int, nz: int, seed: int):
    """A beam on a tilted facet of glass: several passes per step, mask, reflections."""
    rng = np.random.default_rng([seed, ny, nx])
    d = LAM / (8 if nx == 1 else 6)
    y, x = ((np.arange(n) - n // 2) * d for n in (ny, nx))
    front = nz // 3 + np.round(nz / 3 * (0.8 + 0.4 * rng.random()) * np.arange(ny) / ny).astype(int)
    labels = (np.arange(nz)[:, None] >= front[None, :]).astype(np.int32)
    labels = np.broadcast_to(labels[:, :, None], (nz, ny, nx)).copy()
    beam = np.exp(-((y / (ny * d / 6) - 0.3 * rng.random()) ** 2) + 0.1j * K0 * rng.random() * y)[:, None]
    mask = np.exp(-((y / (0.45 * ny * d)) ** 8))[:, None] * np.ones((1, nx))
    if nx > 1:
        beam = beam * np.exp(-((x / (nx * d / 6)) ** 2))[None, :]
        mask = mask * np.exp(-((x / (0.45 * nx * d)) ** 8))[None, :]
    field = np.zeros((ny, nx, 2), complex)
    field[..., 0], field[..., 1] = beam, 0.5j * rng.random() * beam
    index = np.array([1.0, 1.45 + 0.1 * rng.random() + 0j])
    return (ny, nx, d, d if nx > 1 else 1.0, LAM / 10, K0, index, labels, 1.0 + 0j, mask, 0), field


def _ratios_c64(monkeypatch, switch: str, older: str, sizes, nz: int, seeds: int):
    from bwpm_b200 import _core

    logs = []
    for ny, nx in sizes:
        for seed in range(seeds):
            args, field = _volume(ny, nx, nz, seed)
            errors = []
            monkeypatch.delenv(switch, raising=False)
            exact = _core.CudaSolver(*args).run(field, 1, [])
            for mode in ("", older):
                monkeypatch.setenv(switch, mode)
                got = _core.CudaSolver(*args, precision=32).run(field, 1, [])
                errors.append([rel_l2(got[k], exact[k]) for k in ("transmitted", "reflected")])
            logs.extend(np.log(np.array(errors[0]) / np.array(errors[1])))
    return np.array(logs)


def _no_less_exact(logs) -> None:
    bound = 2 * np.std(logs, ddof=1) / np.sqrt(len(logs))
    assert np.mean(logs) <= bound, (float(np.exp(np.mean(logs))), float(bound))


@pytest.mark.parametrize("sizes", [(1200, 2000, 2160, 2688, 3000, 3600),  # run-time lengths over a cluster
                                   (2048, 3072, 4096, 6144, 8192),        # compiled ones
                                   (180, 300, 500, 540, 675, 972)])       # run-time lengths on one CTA
def test_lines_complex64(monkeypatch, sizes):
    _no_less_exact(_ratios_c64(monkeypatch, "BWPM_2D_KERNELS", "step", [(n, 1) for n in sizes], 60, 16))


def test_planes_complex64(monkeypatch):
    _no_less_exact(_ratios_c64(monkeypatch, "BWPM_3D_KERNELS", "general",
                               [(n, n) for n in (180, 300, 400, 432, 500, 540)], 30, 4))


def test_lines_fp64(monkeypatch):
    from bwpm_b200 import _core

    ld = np.longdouble
    steps, index, logs = 60, 1.5, []
    d, dz = LAM / 8, LAM / 10
    for ny in (300, 375, 500, 600, 675, 1875, 2250, 3000, 4050):
        y = (np.arange(ny) - ny // 2) * d
        order = np.arange(ny)
        order[(ny + 1) // 2:] -= ny
        ky = ld("6.283185307179586476925") * order.astype(ld) / (ld(ny) * ld(d))
        kz = np.sqrt(((ld(index) * ld(K0)) ** 2 - ky**2).astype(np.clongdouble))
        args = (ny, 1, d, 1.0, dz, K0, np.array([index + 0j]), np.zeros((steps, ny, 1), np.int32),
                index + 0j, np.ones((ny, 1)), 0)
        solvers = []
        for mode in ("", "step"):
            monkeypatch.setenv("BWPM_2D_KERNELS", mode)
            solvers.append(_core.CudaSolver(*args))
        for seed in range(8):
            rng = np.random.default_rng([seed, ny])
            field = np.zeros((ny, 1, 2), complex)
            field[:, 0, 0] = np.exp(-((y / (ny * d / 8) - 0.5 * rng.random()) ** 2)
                                    + 0.1j * K0 * rng.random() * y)
            spectrum = np.fft.fft(field[:, 0, 0].astype(np.clongdouble))
            exact = np.fft.ifft(spectrum * np.exp(1j * kz * ld(dz) * steps)).astype(complex)
            errors = [rel_l2(s.run(field, 0, [])["transmitted"][:, 0, 0], exact) for s in solvers]
            logs.append(np.log(errors[0] / errors[1]))
    _no_less_exact(np.array(logs))
