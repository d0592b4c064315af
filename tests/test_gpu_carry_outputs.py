"""The step's carry outputs that are formed where the caller wants them (the
saves, muts, muave, mudf, ph_tend, the stage omega) whatever arrays the caller
hands over: left out, shared between outputs nobody wants, placed over an input
that is no longer needed, mudf in place, and a buffer shared by the members of
a batch.  The state must be the ordinary call's bit for bit, and a shared
buffer holds the output that is copied last."""

from __future__ import annotations

import pytest
import torch

from tests import parity_util as P
from wrf_gpu_b200 import cases, dycore

pytestmark = pytest.mark.gpu

# the order in which outputs that share memory are copied out
ORDER = ("mudf", "muave", "muts", "ph_tend", "u_save", "v_save", "w_save", "ph_save", "mu_save", "ww_save")


def _case(kind):
    if kind == "cadence":
        case = cases.real_like_moist(33, 21, 12, hmax=800.0, specified=True, bdy_noise=True)
        case.controls.update(specified_bdy_cadence=True)
        return case
    return cases.real_like_moist(33, 21, 12, hmax=800.0, specified=kind == "specified")


def _step(case, change=None, lead=0.0):
    """One step; ``change(carry, out)`` replaces arrays of the two carries first."""
    stp = dycore.Stepper(dycore.OperationalNamelist.from_case(case))
    carry = dycore.carry_from_case(case)
    carry.mudf = 0.01 * torch.arange(carry.mudf.numel(), dtype=torch.float64, device="cuda").reshape(carry.mudf.shape)
    out = stp.alloc_carry(carry)
    if change is not None:
        change(carry, out)
    stp.step_into(carry, out, lead_seconds=lead)
    torch.cuda.synchronize()
    return out


def _same(ref, got, carry=()):
    for f in P.STATE_KEYS:
        if getattr(ref.state, f) is not None:
            assert torch.equal(getattr(ref.state, f), getattr(got.state, f)), f
    for f in carry:
        assert torch.equal(getattr(ref, f), getattr(got, f)), f


@pytest.mark.parametrize("kind", ["periodic", "specified", "cadence"])
@pytest.mark.parametrize("left_out", [tuple(P.CARRY_KEYS), ORDER, ORDER[::2], ORDER[1::2], ("ww_save",), ("mudf",),
                                      ("u_save", "mu_save"), ("t_2ave", "ww", "t_save")])
def test_left_out(cuda_ready, kind, left_out):
    case = _case(kind)
    got = _step(case, lambda c, o: [setattr(o, f, None) for f in left_out])
    _same(_step(case), got, [f for f in P.CARRY_KEYS if f not in left_out])


@pytest.mark.parametrize("kind", ["periodic", "specified", "cadence"])
def test_outputs_that_share_a_buffer(cuda_ready, kind):
    case = _case(kind)
    flat, faces = ("mudf", "muave", "muts", "mu_save"), ("ph_tend", "w_save", "ph_save", "ww_save")

    def share(carry, out):
        for group in (flat, faces):
            for f in group[1:]:
                setattr(out, f, getattr(out, group[0]))

    ref, got = _step(case), _step(case, share)
    _same(ref, got, [f for f in P.CARRY_KEYS if f not in flat + faces] + ["mu_save", "ww_save"])


@pytest.mark.parametrize("kind", ["periodic", "specified", "cadence"])
def test_saves_over_the_input_state(cuda_ready, kind):
    case = _case(kind)

    def over(carry, out):
        out.u_save, out.v_save, out.w_save = carry.state.u, carry.state.v, carry.state.w
        out.ph_save, out.mu_save = carry.state.ph_perturbation, carry.state.mu_perturbation
        out.muts, out.ww_save = carry.state.mu_total, carry.state.ph_total

    _same(_step(case), _step(case, over), P.CARRY_KEYS)


def test_partly_shared(cuda_ready):
    """Two face outputs one level apart in one allocation."""
    case = _case("periodic")

    def share(carry, out):
        nl, ny, nx = out.w_save.shape
        pool = torch.empty((nl + 1, ny, nx), dtype=torch.float64, device="cuda")
        out.w_save, out.ww_save = pool[:nl], pool[1:]

    ref, got = _step(case), _step(case, share)
    _same(ref, got, [f for f in P.CARRY_KEYS if f != "w_save"])
    assert torch.equal(ref.w_save[0], got.w_save[0])


@pytest.mark.parametrize("kind", ["periodic", "specified"])
def test_mudf_in_place(cuda_ready, kind):
    case = _case(kind)
    _same(_step(case), _step(case, lambda c, o: setattr(o, "mudf", c.mudf)), P.CARRY_KEYS)


def test_members_of_a_batch_share_a_buffer(cuda_ready):
    cs = [_case("periodic"), _case("specified")]
    nls = [dycore.OperationalNamelist.from_case(c) for c in cs]
    bs = dycore.BatchStepper(nls)
    carries = [dycore.carry_from_case(c) for c in cs]
    outs = bs.alloc_carries(carries)
    for f in ("w_save", "ph_save", "mu_save"):
        setattr(outs[1], f, getattr(outs[0], f))
    bs.step_into(carries, outs, lead_seconds=0.0)
    torch.cuda.synchronize()
    for nl, c, got in zip(nls, carries, outs):
        ref = dycore.rk_scan_step(c, nl, lead_seconds=0.0)
        _same(ref, got, [f for f in P.CARRY_KEYS if f not in ("w_save", "ph_save", "mu_save")])
