"""The top-face extrapolation weights formed on the device (``cfn`` = NaN in the
params, the Python shim's default) against the same weights handed in by the
caller, bit for bit: the rigid lid's pressure gradient (stretched levels) and
the order-6 rhs_ph's open top; and no step call waits for the GPU for them."""

from __future__ import annotations

import math

import pytest
import torch

from tests import parity_util as P
from wrf_gpu_b200 import cases, dycore

pytestmark = pytest.mark.gpu


def _case(kind):
    case = cases.mountain_wave(28, 24, 16)
    if kind == "lid":
        case.controls.update(top_lid=True)
    else:
        case.controls.update(h_sca_adv_order=5)
    return case


@pytest.mark.parametrize("kind", ["lid", "open_order6"])
def test_device_weights_match_the_callers(cuda_ready, kind):
    case = _case(kind)
    nl = dycore.OperationalNamelist.from_case(case)
    carry = dycore.carry_from_case(case)
    outs = []
    for given in (False, True):
        st = dycore.Stepper(nl)
        assert math.isnan(st.params.cfn)
        if given:
            st.params.cfn, st.params.cfn1 = nl.metrics.cfn()
        out = st.alloc_carry(carry)
        st.step_into(carry, out, lead_seconds=0.0)
        outs.append(out)
    torch.cuda.synchronize()
    for k in P.STATE_KEYS:
        assert torch.equal(getattr(outs[0].state, k), getattr(outs[1].state, k)), k
    for k in P.CARRY_KEYS:
        assert torch.equal(getattr(outs[0], k), getattr(outs[1], k)), k


def test_the_step_call_does_not_synchronise(cuda_ready):
    case = _case("lid")
    nl = dycore.OperationalNamelist.from_case(case)
    carry = dycore.carry_from_case(case)
    dycore.rk_scan_step(carry, nl, lead_seconds=0.0)
    torch.cuda.synchronize()
    torch.cuda.set_sync_debug_mode("error")
    try:
        dycore.rk_scan_step(carry, nl, lead_seconds=0.0)
    finally:
        torch.cuda.set_sync_debug_mode("default")
    torch.cuda.synchronize()
