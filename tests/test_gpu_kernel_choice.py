"""That the kernels which the size tests are about are the ones that run, on a GPU.

A size without a one-launch or register-resident kernel takes the older kernels without a word, and
their results are the same but for rounding. So the choice is read off what tells the forms apart:
the launches of a run and the device bytes a solver holds. Of the sizes of test_gpu_chain2d.py,
test_gpu_born2d.py and test_gpu_plane_sizes.py those are left out that keep the older kernels: 210
points (no E² divides them), FP64 Born lines of 2430 and 6144 points and complex64 ones other than
512, 1024 and 4096, planes with a side of 2187 points, in FP64 of 1600.
"""

from __future__ import annotations

import pytest

from test_gpu_solver_sharing import _case, _line, _plane

pytestmark = pytest.mark.gpu


def _launches(args, kw, field, precision):
    from bwpm_b200 import _core

    s = _core.CudaSolver(*args, 0, precision=precision, **kw)
    s.run(field, 1, [])  # the first run also builds tables
    before = s.stats()["kernel_launches"]
    s.run(field, 1, [])
    return s.stats()["kernel_launches"] - before


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("masked", [True, False])
@pytest.mark.parametrize("ny", [4, 18, 150, 256, 343, 375, 384, 512, 768, 1024, 1080, 1500, 1536, 1944, 2048,
                                2187, 2430, 2500, 3072, 3600, 4050, 4096, 5120, 6144, 8192])
def test_chain_kernel_runs(monkeypatch, ny, masked, precision):
    """A run is one launch beside the conversions of its planes."""
    monkeypatch.delenv("BWPM_2D_KERNELS", raising=False)
    args, field = _line(ny, 24, masked)
    assert _launches(args, {}, field, precision) <= 8


@pytest.mark.parametrize("precision,ny", [(64, n) for n in (64, 144, 250, 512, 640, 1000, 1024, 1536, 2048, 3072,
                                                            3584, 4096)]
                         + [(32, n) for n in (512, 1024, 4096)])
def test_born_kernel_runs(monkeypatch, ny, precision):
    """A slab is its step and one launch per direction; the multi-kernel form launches its
    transforms, sources and emissions one by one around each graph."""
    args, field, kw = _case("born", ny)
    monkeypatch.delenv("BWPM_GMRES", raising=False)
    one = _launches(args, kw, field, precision)
    monkeypatch.setenv("BWPM_GMRES", "graph")
    assert 2 * one < _launches(args, kw, field, precision)


@pytest.mark.parametrize("precision,ny,nx",
                         [(p, ny, nx) for p in (64, 32)
                          for ny, nx in ((4, 8), (9, 4), (16, 36), (49, 50), (45, 36), (64, 256), (243, 125),
                                         (375, 250), (256, 384), (384, 100), (768, 18), (18, 1024), (300, 512),
                                         (98, 27), (512, 768), (1024, 1024))] + [(32, 1600, 16)])
def test_plane_kernels_run(monkeypatch, precision, ny, nx):
    """Their operator tables hold a quarter plane."""
    from bwpm_b200 import _core

    args, field = _plane(ny, nx, 4)
    held = {}
    for kernels in ("", "general"):
        monkeypatch.setenv("BWPM_3D_KERNELS", kernels)
        s = _core.CudaSolver(*args, 0, precision=precision)
        s.run(field, 1, [])
        held[kernels] = s.stats()["device_bytes"]
    assert held[""] < held["general"]
