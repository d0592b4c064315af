"""The one-thread-per-column acoustic column kernel (``k_column_stream``,
selected by ``column_width = 1``) against the level-parallel one
(``k_column_tiled``, widths 16 / 32): the whole RK3 step must come out bit
for bit identical, on every branch the column kernel has -- periodic and
specified columns, the boundary cadence's and the nested child's ring-0 pins,
w damping, Rayleigh damping, the rigid lid, grids off every 32-column and
4-row multiple and a one-column slab."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests import parity_util as P
from wrf_gpu_b200 import cases, dycore

pytestmark = pytest.mark.gpu


def _step(case, width, lead=0.0, lanes=0):
    nl = dycore.OperationalNamelist.from_case(case)
    stp = dycore.Stepper(nl)
    stp.params.column_width, stp.params.column_lanes = width, lanes
    a = dycore.carry_from_case(case)
    b = stp.alloc_carry(a)
    stp.step_into(a, b, lead_seconds=lead)
    torch.cuda.synchronize()
    return b


def _variants():
    out = []
    out.append(("periodic", cases.real_like_moist(37, 21, 14, hmax=800.0, specified=False)))
    out.append(("specified", cases.real_like_moist(45, 19, 14, hmax=800.0, specified=True)))
    c = cases.real_like_moist(40, 24, 12, hmax=800.0, specified=True, bdy_noise=True)
    c.controls.update(specified_bdy_cadence=True)
    out.append(("cadence", c))
    c = cases.real_like_moist(40, 24, 12, hmax=800.0, specified=True, bdy_noise=True)
    c.controls.update(force_geopotential=False, nested_ph_relax=True, nested_ph_spec=True)
    out.append(("nested", c))
    c = cases.real_like_moist(33, 17, 12, hmax=600.0, specified=False)
    c.controls.update(w_damping=1, damp_opt=3, dampcoef=0.2, zdamp=5000.0)
    out.append(("damping", c))
    c = cases.real_like_moist(33, 17, 12, hmax=600.0, specified=False)
    c.controls.update(top_lid=True)
    out.append(("top_lid", c))
    out.append(("mountain_wave", cases.mountain_wave(28, 24, 16)))
    out.append(("slab", cases.real_like_moist(1, 6, 5, hmax=300.0, specified=False)))
    out.append(("warm_bubble", cases.warm_bubble_3d(20, 16, 12)))
    return out


@pytest.mark.parametrize("name,case", _variants(), ids=[v[0] for v in _variants()])
def test_stream_column_kernel_is_bit_identical(cuda_ready, name, case):
    ref = _step(case, 32)
    for width in (1, 16):
        got = _step(case, width)
        for f in P.STATE_KEYS:
            a, b = getattr(ref.state, f), getattr(got.state, f)
            if a is None:
                continue
            assert torch.equal(a, b), (name, width, f, float((a - b).abs().max()))
        for f in P.CARRY_KEYS:
            assert torch.equal(getattr(ref, f), getattr(got, f)), (name, width, f)


def _tall(nz, kind):
    if kind in ("cadence", "nested"):
        c = cases.real_like_moist(21, 12, nz, hmax=800.0, specified=True, bdy_noise=True)
        c.controls.update(**(dict(specified_bdy_cadence=True) if kind == "cadence" else
                             dict(force_geopotential=False, nested_ph_relax=True, nested_ph_spec=True)))
        return c
    c = cases.real_like_moist(19, 11, nz, hmax=600.0, specified=kind == "specified")
    if kind == "damping":
        c.controls.update(w_damping=1, damp_opt=3, dampcoef=0.2, zdamp=5000.0)
    if kind == "top_lid":
        c.controls.update(top_lid=True)
    return c


# heights on both sides of every change in the number of levels per lane (52 |
# 53 and 78 | 79 faces by default; 34 | 35 with 17 lanes, 53 with 13), and lane
# counts that the height sends to the default
@pytest.mark.parametrize("kind", ["specified", "cadence", "nested", "damping", "top_lid"])
@pytest.mark.parametrize("nz,lanes", [(51, 0), (52, 0), (77, 0), (78, 0), (95, 0), (33, 17), (34, 17), (51, 13),
                                      (52, 13), (50, 8), (70, 16)])
def test_every_position_count_is_bit_identical_on_every_branch(cuda_ready, nz, lanes, kind):
    case = _tall(nz, kind)
    ref = _step(case, 1)
    for width in (16, 32):
        got = _step(case, width, lanes=lanes)
        for f in P.STATE_KEYS:
            if getattr(ref.state, f) is not None:
                assert torch.equal(getattr(ref.state, f), getattr(got.state, f)), (width, f)
        for f in P.CARRY_KEYS:
            assert torch.equal(getattr(ref, f), getattr(got, f)), (width, f)
