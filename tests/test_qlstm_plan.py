"""The plan of a QLstm layer: which input magnitudes can bring a product close to a rounding boundary."""
import ctypes as C
import time

import numpy as np
import pytest

from armnn_b200 import _abi, lib
from q8util import Cuda, diff_stats, random_qlstm_case


def _params(**scales):
    """A layer without weights' contents: the plan depends on its scales and on which weights there are."""
    p = _abi.QLstmParams()
    p.w_i2i = p.w_i2f = p.w_i2c = p.w_i2o = p.w_r2i = p.w_r2f = p.w_r2c = p.w_r2o = p.w_proj = 1
    p.input_scale, p.output_state_scale, p.hidden_state_scale, p.output_scale, p.s_proj = 1 / 128, 0.007, 0.0065, 0.0071, 1 / 255
    for k, g in enumerate("ifco"):
        setattr(p, "s_i2" + g, 0.0078 + 0.0003 * k)
        setattr(p, "s_r2" + g, 0.0039 + 0.0002 * k)
    p.input_intermediate_scale = p.cell_intermediate_scale = 0.007059
    p.forget_intermediate_scale = p.output_intermediate_scale = 0.007812
    for k, v in scales.items():
        setattr(p, k, v)
    return p


def _near_half(sx, sw, sg):
    c = float(np.float32(sx)) * float(np.float32(sw)) / float(np.float32(sg))
    r = (np.arange(256)[:, None] * np.arange(129)[None, :]).astype(np.float64) * c
    return (np.abs(r - np.floor(r) - 0.5) <= (8 * r + 8 + 3 * 2048) * 2.0 ** -24).any(1)


def _magnitudes(plan, source, pair):
    return np.unpackbits(np.asarray(plan.magnitudes[source][pair], dtype="<u4").view(np.uint8), bitorder="little").astype(bool)


@pytest.mark.parametrize("scales", [{}, dict(input_scale=2.0 ** -7, s_i2f=2.0 ** -7, forget_intermediate_scale=2.0 ** -13), dict(s_r2o=300.0, output_scale=1e-7), dict(w_i2i=None),
                                    dict(s_i2c=2.0 ** -9, input_scale=0.5, cell_intermediate_scale=0.25)],
                         ids=["plain", "halves", "large_quotients", "cifg", "powers_of_two"])
def test_plan_lists_the_magnitudes_near_a_half(scales):
    p, plan = _params(**scales), _abi.QLstmPlan()
    lib.check(lib.load_library().b200k_qlstm_prepare(C.byref(p), C.byref(plan)))
    first = "f" if p.w_i2i is None else "i"
    gates = [(first, p.forget_intermediate_scale if first == "f" else p.input_intermediate_scale), ("f", p.forget_intermediate_scale),
             ("c", p.cell_intermediate_scale), ("o", p.output_intermediate_scale)]
    for pair in (0, 1):
        for source, sx, prefix in ((0, p.input_scale, "s_i2"), (1, p.output_state_scale, "s_r2")):
            want = np.zeros(256, bool)
            for g, sg in gates[pair::2]:
                want |= _near_half(sx, getattr(p, prefix + g), sg)
            assert np.array_equal(_magnitudes(plan, source, pair)[1:], want[1:]), (source, pair)
    assert np.array_equal(_magnitudes(plan, 2, 0)[1:], _near_half(p.hidden_state_scale, p.s_proj, p.output_scale)[1:])


def test_plan_of_scales_that_the_bound_does_not_hold_for_is_empty():
    p, plan = _params(input_scale=1e-9), _abi.QLstmPlan()
    lib.check(lib.load_library().b200k_qlstm_prepare(C.byref(p), C.byref(plan)))
    assert not any(_magnitudes(plan, s, g).any() for s in range(3) for g in range(2))
    assert lib.load_library().b200k_qlstm_prepare(None, C.byref(plan)) == _abi.E_INVALID


@pytest.mark.gpu
def test_a_plan_is_used_for_its_own_scales_only(built):
    """With its plan, without one, and with another layer's: the same step.  2^-7 scales make every product a multiple of a half."""
    case = random_qlstm_case(3, 5, 48, 40, 24)
    for g in "ifco":
        case.s["s_i2" + g] = case.s["s_r2" + g] = 2.0 ** -7
    for g in ("input", "forget", "cell", "output"):
        case.s[g + "_intermediate_scale"] = 2.0 ** -7
    want = case.run_oracle()
    l = lib.load_library()
    other = _abi.QLstmPlan()
    lib.check(l.b200k_qlstm_prepare(C.byref(_params()), C.byref(other)))
    got = []
    for which in ("own", None, "other"):
        mem = Cuda()
        p, outs = case.params(mem)
        own = _abi.QLstmPlan()
        lib.check(l.b200k_qlstm_prepare(C.byref(p), C.byref(own)))
        if which:
            p.plan = C.pointer(own if which == "own" else other)
        lib.call("qlstm_step", p)
        got.append([mem.fetch(o) for o in outs])
    for g in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got[0], g))
    for w, g in zip(want, got[0]):
        st = diff_stats(w, g)                  # (exp and tanh: see test_shape_edges_gpu.py)
        assert st["max_abs"] <= (2 if w.dtype == np.int16 else 1) and st["mismatch_frac"] <= 0.01, st


@pytest.mark.gpu
@pytest.mark.parametrize("layers", [10, 40])
def test_stepping_many_layers_with_scales_of_their_own_costs_no_planning(built, layers):
    """Host time of a stack's steps from the second pass on: the launches, not the planning (0.4 ms a layer)."""
    calls, keep = [], []
    for i in range(layers):
        case = random_qlstm_case(i, 1, 16, 16, 16)
        for j, k in enumerate(k for k in case.s if "scale" in k or k.startswith(("s_i2", "s_r2", "s_proj"))):
            case.s[k] = float(np.float32(case.s[k] * (1 + 0.0003 * (37 * i + j))))
        mem = Cuda()
        p, _ = case.params(mem)
        keep.append((mem, case))
        calls.append(p)
    l = lib.load_library()
    mem.torch.cuda.synchronize()
    seconds = []
    for _ in range(5):
        t = time.perf_counter()
        for p in calls:
            lib.check(l.b200k_qlstm_step(C.byref(p), None))
        seconds.append(time.perf_counter() - t)
        mem.torch.cuda.synchronize()
    assert min(seconds[1:]) / layers < 1.5e-4, seconds
