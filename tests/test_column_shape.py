"""The acoustic column kernels' launch shape (``csrc/column_shape.cuh``, host
arithmetic) for every height, width and lane count the params accept, compiled
here with the default column width of the build and with each of the others:
a width of 1 -- asked for or the default -- is the streaming kernel, every
level-parallel block covers its levels within the kernel's bounds, and no
request gets more than four positions per lane, where the kernel is slow."""

from __future__ import annotations

import shutil
import subprocess

import pytest

from wrf_gpu_b200 import build

PROGRAM = """
#include <cstdio>
#include <initializer_list>
#include "column_shape.cuh"
int main() {
  for (int nz = 4; nz <= 130; ++nz)
    for (int w : {0, 1, 16, 32})
      for (int l : {0, 8, 13, 16, 17}) {
        const wg::ColumnShape s = wg::column_shape(nz, w, l);
        std::printf("%d %d %d %d %d %d %d %zu %d\\n", nz, w, l, s.stream, s.tx, s.ty, s.np, s.smem, s.too_tall);
      }
  for (int nz = 4; nz <= 112; ++nz) {
    wg::ColumnRequest c[wg::COL_MAX_CANDIDATES];
    const int n = wg::column_candidates(nz, c);
    std::printf("candidates %d", nz);
    for (int k = 0; k < n; ++k) std::printf(" %d %d", c[k].width, c[k].lanes);
    std::printf("\\n");
  }
  std::printf("%d %d %d\\n", wg::COL_TY, wg::COL_MAX_NZ, wg::CS_WARPS);
}
"""
SMEM_PER_BLOCK = 227 * 1024


def _shapes(tmp_path, default):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "shape.cc", tmp_path / "shape"
    src.write_text(PROGRAM)
    flags = [f"-DWG_COL_DEFAULT_WIDTH={default}"] if default else []
    subprocess.run([gxx, "-std=c++17", *flags, "-I", str(build.CSRC), "-o", str(exe), str(src)], check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    ints = lambda line: tuple(map(int, line.split()))
    tuner = [ints(line[len("candidates"):]) for line in lines if line.startswith("candidates")]
    rows = [ints(line) for line in lines if not line.startswith("candidates")]
    return rows[:-1], rows[-1], {t[0]: list(zip(t[1::2], t[2::2])) for t in tuner}


@pytest.mark.parametrize("default", [None, 1, 16, 32])
def test_every_accepted_shape(tmp_path, default):
    rows, (max_lanes, max_nz, stream_warps), _ = _shapes(tmp_path, default)
    for nz, width, lanes, stream, tx, ty, np_, smem, too_tall in rows:
        what = (default, nz, width, lanes)
        wanted = width or default or 16
        assert bool(stream) == (wanted == 1), what
        if stream:
            assert (tx, ty, too_tall) == (32, stream_warps, 0), what
            assert smem == 2 * (nz + 1) * 32 * stream_warps * 8, what
            continue
        assert tx == wanted and bool(too_tall) == (nz > max_nz), what
        if too_tall:
            continue
        # warp 0 is left to the serial phases, the next one forms the surface w
        assert 32 // tx + 1 <= ty <= max_lanes, what
        assert ty * np_ >= nz + 1, what
        # positions: those of the lanes asked for up to four, else the built-in count's
        default_np = max(2, -(-(nz + 1) // max_lanes))
        asked = -(-(nz + 1) // lanes) if lanes else default_np
        assert np_ == max(2, asked if asked <= 4 else default_np), what
        assert 2 <= np_ <= (4 if nz < 4 * max_lanes else 5), what
        # eight level arrays, and the level coefficients where they are staged
        assert smem >= 8 * tx * (nz + 1) * 8 and smem + 4 * tx * 8 <= SMEM_PER_BLOCK, what


def test_the_tuner_times_no_launch_twice(tmp_path):
    rows, _, tuner = _shapes(tmp_path, None)
    launch = {r[:3]: r[3:7] for r in rows}
    for nz, cands in tuner.items():
        launches = [launch[nz, w, lanes] for w, lanes in cands]
        assert len(set(launches)) == len(launches), (nz, cands)
        # nothing that 17 or 13 lanes would give is missed
        assert set(launches) == {launch[nz, w, lanes] for w in (1, 16, 32) for lanes in (0, 17, 13)}, (nz, cands)
    assert tuner[50] == [(16, 0), (16, 17), (16, 13), (32, 0), (32, 17), (32, 13), (1, 0)]
    assert tuner[20] == [(16, 0), (32, 0), (1, 0)]
