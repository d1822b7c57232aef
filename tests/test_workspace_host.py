"""Sizes of the adjoint workspaces (host functions, no GPU): a call asks for what its plan and
variables can use -- a block of 256 rays in the fused adjoint (128 in plans of at most 3,072 rays)
keeps (columns + 10 S) values per ray and two sums of its tile pairs, a block of 128 rays of the
Jacobian 10 S + 1 -- and the sizes that are asked for without a plan suit every plan."""

import ctypes as C
import dataclasses

import pytest

from mikroptim_b200 import _capi, workloads
from mikroptim_b200.batch import (PRECISION_FP64, PRECISION_MIXED, ResidualLayout)
from mikroptim_b200.engine import LmOptions, TraceEngine, JACOBIAN_ADJOINT

SMS = 148


def _case(make, precision, **kw):
    b, st, vs, x0 = make(2, **kw)
    lay = ResidualLayout(b.topology, dataclasses.replace(st, precision=precision))
    shape = TraceEngine._shape(b.topology, b.buchdahl_coeff is not None)
    shape.variants = 1
    shape.records = C.c_void_p(0x10000)  # never dereferenced
    return b, lay.plan(b), shape, vs


def _fused(b, plan, precision):
    """Threads of a block, blocks at most, and the most pieces of a run: whole tuples of at least 192
    rays (plans of few rays) or 512 (but for the last piece)."""
    rays = int(_capi.lib().mkb_rays_per_variant(C.byref(plan)))
    threads = 128 if rays <= 3072 else 256
    mixed = precision == PRECISION_MIXED
    blocks = SMS * ((4 if mixed else 3) if threads == 128 else (2 if mixed else 1))
    return threads, blocks, min(b.fields * b.wavelengths, -(-rays // (192 if threads == 128 else 512)))


def _slot(P, S, precision, threads):
    cols = (P + 8) // 8
    values = (8 * cols + 10 * S) * threads * (4 if precision == PRECISION_MIXED else 8)
    return values, cols * (cols + 1) // 2 * 512


CASES = [
    (workloads.singlet, {}),
    (workloads.sweep, dict(surfaces=30, wavelengths=7, rings=16, spokes=32)),
    (workloads.sweep, dict(surfaces=43, wavelengths=2, rings=3, spokes=5)),
    (workloads.sweep, dict(surfaces=10, wavelengths=7, rings=6, spokes=12)),
]


@pytest.mark.parametrize("make,kw", CASES)
@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_MIXED])
@pytest.mark.parametrize("runs", [1, 4, 48, 400, 5000])
def test_fused_workspace_holds_what_the_items_use(make, kw, precision, runs):
    lib = _capi.lib()
    b, plan, shape, vs = _case(make, precision, **kw)
    threads, ctas, pieces = _fused(b, plan, precision)
    v = vs.c_struct()
    need = int(lib.mkb_adjoint_normal_equations_workspace_bytes(C.byref(shape), C.byref(plan),
                                                                C.byref(v), 0, runs))
    values, sums = _slot(vs.size, b.surfaces, precision, threads)
    assert need >= 8 * runs * shape.record_stride + (values + 2 * sums)  # a block at least
    # records, counters, the items' sums, the blocks' states; three parts are rounded up to 256
    assert need <= (8 * runs * shape.record_stride + 4 * (runs + 64) + 3 * 256 +
                    (min(runs * pieces * sums, 160 << 20) if pieces > 1 else 0) +
                    min(runs * pieces, ctas) * (values + 2 * sums))
    assert need <= int(lib.mkb_adjoint_jacobian_workspace_bytes(C.byref(shape), runs))
    # enough runs to fill the GPU are one item each: no sums
    if runs >= 8 * ctas:
        assert need <= (8 * runs * shape.record_stride + 4 * (runs + 64) + 3 * 256 +
                        ctas * (values + 2 * sums))
    # the LM holds that scratch, its own state and the trial merits
    shape.variants = runs
    opt = LmOptions(jacobian=JACOBIAN_ADJOINT, gram_exact=False).c_struct()
    lm = int(lib.mkb_lm_workspace_bytes(C.byref(shape), C.byref(plan), C.byref(v), C.byref(opt),
                                        runs))
    P = vs.size
    assert need < lm <= need + runs * (8 * (2 * P * P + 8 * P + 400) + 64 * b.fields *
                                       b.wavelengths + 512) + 64 * 256


@pytest.mark.parametrize("make,kw", CASES)
@pytest.mark.parametrize("runs", [1, 4, 48, 400])
def test_jacobian_workspace_holds_the_kept_states(make, kw, runs):
    lib = _capi.lib()
    b, plan, shape, vs = _case(make, PRECISION_FP64, **kw)
    blocks = runs * -(-int(lib.mkb_rays_per_variant(C.byref(plan))) // 128)
    need = int(lib.mkb_adjoint_jacobian_plan_workspace_bytes(C.byref(shape), C.byref(plan), runs))
    states = min(blocks, 3 * SMS) * (10 * b.surfaces + 1) * 128 * 8
    assert 0 <= need - (8 * runs * shape.record_stride + states) < 256


def test_no_size_without_a_valid_plan():
    lib = _capi.lib()
    b, plan, shape, vs = _case(workloads.singlet, PRECISION_FP64)
    v = vs.c_struct()
    plan.rings = 0
    assert lib.mkb_adjoint_jacobian_plan_workspace_bytes(C.byref(shape), C.byref(plan), 4) == 0
    assert lib.mkb_adjoint_normal_equations_workspace_bytes(C.byref(shape), C.byref(plan),
                                                            C.byref(v), 0, 4) == 0
    assert lib.mkb_adjoint_normal_equations_workspace_bytes(None, C.byref(plan), C.byref(v), 0,
                                                            4) == 0
