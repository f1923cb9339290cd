"""The 2D chain kernels (bwpm_b200/csrc/chain2d.cuh) on a GPU.

Every sweep of a 2D solve runs in one launch, with compiled lengths (256 … 8192) and run-time
ones, on one CTA or split over a cluster. A volume with three materials (one absorbing), a tilted face, so steps of one
and of several passes, and a planar end goes through the chain kernels and through the
launch-per-step kernels (BWPM_2D_KERNELS=step), and both are held to the numpy oracle: FP64 at
the drop-in contract (1e-10), complex64 at the complex64 contract (relative L2 ≤ 1e-4). Without a
mask, runs of single-pair steps stay in the spectrum; kept planes and sources interrupt them.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = {64: 1e-10, 32: 1e-4}


def _case(ny: int, nz: int, masked: bool):
    rng = np.random.default_rng(ny)
    lam = 0.633e-3
    dy, dz = lam / 8, lam / 10
    y = (np.arange(ny) - ny // 2) * dy
    labels = np.zeros((nz, ny), np.int32)
    front = 3 + np.round(3 * (y - y[0]) / (ny * dy)).astype(int)  # crosses slabs 3 … 6
    for j in range(nz):
        labels[j, j >= front] = 1
    labels[nz - 3:] = 2  # planar back face: a step of one pair with reflections
    field = np.zeros((ny, 1, 2), complex)
    beam = np.exp(-((y / (ny * dy / 5)) ** 2) + 0.3j * y / dy)
    field[:, 0, 0] = beam
    field[:, 0, 1] = 0.4j * beam * rng.uniform(0.9, 1.1, ny)
    mask = np.exp(-((y / (0.45 * ny * dy)) ** 8))[:, None] if masked else None
    args = (ny, 1, dy, 1.0, dz, 2 * np.pi / lam, np.array([1.0, 1.5, 1.2 + 0.05j]),
            labels[:, :, None], 1.0 + 0j, mask)
    return args, field


@pytest.mark.parametrize("masked", [True, False])
@pytest.mark.parametrize("ny", [4, 18, 150, 210, 256, 343, 375, 384, 512, 768, 1024, 1080, 1500, 1536, 1944,
                                2048, 2187, 2430, 2500, 3072, 3600, 4050, 4096, 5120, 6144, 8192])
def test_chain_matches_step_kernels_and_oracle(monkeypatch, ny, masked):
    from bwpm_b200 import _core
    from oracle import port

    nz, iters, keep = 14, 2, [0, 2, 5, 13, 14]
    args, field = _case(ny, nz, masked)
    ref = port.Solver(*args).run(field, iters, keep)
    ref0 = port.Solver(*args).run(field, 0, [])
    for prec in (64, 32):
        for mode in ("chain", "step"):
            monkeypatch.setenv("BWPM_2D_KERNELS", mode)
            s = _core.CudaSolver(*args, 0, precision=prec)
            for got, want, keys in ((s.run(field, iters, keep), ref, ("transmitted", "reflected")),
                                    (s.run(field, 0, []), ref0, ("transmitted",)),
                                    (s.run(field, iters, []), ref, ("transmitted", "reflected"))):
                for key in keys:
                    assert rel_l2(got[key], want[key]) < TOL[prec], (prec, mode, key)
            got = s.run(field, iters, keep)
            for q in keep:
                assert rel_l2(got["forward"][q], ref["forward"][q]) < TOL[prec], (prec, mode, q)
                if q < nz:  # the backward sweep starts from a zero plane
                    assert rel_l2(got["backward"][q], ref["backward"][q]) < TOL[prec], (prec, mode, q)
                else:
                    assert not np.any(got["backward"][q])
            for it in range(iters):
                assert np.all(np.isfinite(got["transmitted_iter"][it]))
            assert np.array_equal(got["transmitted_iter"][-1], got["transmitted"])
