"""Kernels whose level split is chosen from the grid, against the oracle.

``advance_uv`` marches 1 to 17 levels per thread and the column kernel holds 2
or more levels per lane, both picked from the grid's size: one step at grids on
either side of the choices (a chunk of one level, a short last chunk, the
longest chunks; two, three and four levels per lane)."""

from __future__ import annotations

import pytest

from tests.test_gpu_parity import _per_step
from wrf_gpu_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(5, 3, 4), (33, 9, 5), (24, 20, 53), (18, 7, 79), (9, 8, 95), (420, 200, 19)])
def test_step_matches_oracle_for_every_level_split(cuda_ready, nx, ny, nz):
    case = cases.real_like_moist(nx, ny, nz, hmax=300.0, specified=False)
    # the step starts from w = 0: w and the mass diagnostics of its first step
    # are at the noise floor, where one-ulp pow() differences of the oracle
    # reach 1.7e-12 relative at 53 levels; a wrong split is an error of order 1
    for k, e in _per_step(case, 1)[0].items():
        assert e <= 1.0e-10, (k, e)
