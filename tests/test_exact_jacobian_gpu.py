"""The bit-exact Jacobian path at the edges of its tiles: the normal equations' chains (gram.cu:
16-column tiles, 32-row stages), the rows from kept states (adjoint.cu: 128-ray chunks) and the
piston projection (64-sample tiles), each equal to the oracle bit for bit."""

import numpy as np
import pytest
import torch

from mikroptim_b200 import engine, workloads
from mikroptim_b200.batch import FAILURE_HARD, FAILURE_SOFT, ResidualLayout
import oracle.pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 7, 15, 16, 31, 47, 64])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 128, 197])
def test_chains_equal_the_oracle(P, rows):
    rng = np.random.default_rng(100 * P + rows)
    J, r = rng.normal(size=(3, P, rows)), rng.normal(size=(3, rows))
    J[:, :, rows // 2] = -0.0
    got = engine.normal_equations_device(torch.from_numpy(J).cuda(), torch.from_numpy(r).cuda(),
                                         True).cpu().numpy()
    for i in range(3):
        A, g = po.port().normal_equations(J[i], r[i])
        assert np.array_equal(got[i, :P, :P], A) and np.array_equal(got[i, :P, P], g)
        assert np.array_equal(got[i], got[i].T)


@pytest.mark.parametrize("P", [2, 6, 8, 17, 18, 19, 20, 23, 34, 35, 36, 50])
@pytest.mark.parametrize("rows", [35, 96, 100])
def test_chains_of_narrow_and_last_tiles_equal_the_oracle(P, rows):
    """One chain per thread up to eight columns; one to four columns in the last tile of sixteen,
    whose own chains the pair with the first tile takes, and five."""
    test_chains_equal_the_oracle(P, rows)


@pytest.mark.parametrize("P", [1, 4, 7, 8])
@pytest.mark.parametrize("rows", [1, 3, 127, 128, 129, 900])
def test_tensor_core_sums_of_few_columns(P, rows):
    """Eight columns or fewer take one tile without staging. A sum of n products is within
    n 2^-53 sum |a b| of the exact one in any order."""
    rng = np.random.default_rng(100 * P + rows)
    J, r = rng.normal(size=(3, P, rows)), rng.normal(size=(3, rows))
    got = engine.normal_equations_device(torch.from_numpy(J).cuda(), torch.from_numpy(r).cuda(),
                                         False).cpu().numpy()
    X = np.concatenate([J, r[:, None]], axis=1).astype(np.longdouble)
    want = X @ X.transpose(0, 2, 1)
    bound = (rows + 1) * 2.0 ** -53 * (np.abs(X) @ np.abs(X).transpose(0, 2, 1))
    assert (np.abs(got - want) <= bound).all()
    assert np.array_equal(got, got.transpose(0, 2, 1))


@pytest.mark.parametrize("failure", [FAILURE_SOFT, FAILURE_HARD])
@pytest.mark.parametrize("rings,spokes,glass", [
    (1, 1, False),    # 35 rays, tuples of one ray
    (3, 21, True),    # tuples of 63 rays
    (4, 16, False),   # of 64
    (5, 13, True),    # of 65; 7 rays in the last chunk
])
def test_rows_and_projection_equal_the_oracle(rings, spokes, glass, failure):
    b, st, vs, x0 = workloads.objective(5, rings=rings, spokes=spokes, glass=glass,
                                        failure=failure)
    lay = ResidualLayout(b.topology, st)
    J, r, s = engine.adjoint_jacobian_device(engine.DeviceSystemBatch(b), lay, b, vs, x0)
    Jo, ro, so = po.port().adjoint_jacobian(b, lay, vs, x0, threads=8)
    assert np.array_equal(s.cpu().numpy(), so) and np.array_equal(r.cpu().numpy(), ro)
    J = J.cpu().numpy()
    # bit for bit, the signs of zeros included
    assert np.array_equal(J.view(np.int64), Jo.view(np.int64)), np.argwhere(J != Jo)[:5]


def test_fewer_blocks_share_the_workspace_sized_without_a_plan():
    """The size without a plan is below the plan's here: the rows are the same bits, and one byte
    less is refused."""
    import ctypes as C
    from mikroptim_b200 import _capi
    lib = _capi.lib()
    b, st, vs, x0 = workloads.sweep(4, surfaces=30, wavelengths=7, rings=16, spokes=32)
    lay = ResidualLayout(b.topology, st)
    db = engine.DeviceSystemBatch(b)
    J, r, s = engine.adjoint_jacobian_device(db, lay, b, vs, x0)
    t, plan, v = db.c_struct(), lay.plan(b), vs.c_struct()
    need = int(lib.mkb_adjoint_jacobian_workspace_bytes(C.byref(t), 4))
    assert need < int(lib.mkb_adjoint_jacobian_plan_workspace_bytes(C.byref(t), C.byref(plan), 4))
    x = engine._dev_f64(x0, db.device)
    ws = torch.empty(need, dtype=torch.uint8, device=db.device)
    J2, r2, s2 = torch.empty_like(J), torch.empty_like(r), torch.empty_like(s)

    def call(nbytes):
        return lib.mkb_adjoint_jacobian_device(
            C.byref(t), C.byref(plan), C.byref(v), C.c_void_p(x.data_ptr()), 4,
            *(C.c_void_p(a.data_ptr()) for a in (J2, r2, s2, ws)), nbytes, None)
    assert call(need - 1) == _capi.MKB_ERR_WORKSPACE
    torch.cuda.synchronize()
    _capi.check(call(need), "adjoint jacobian")
    torch.cuda.synchronize()
    assert torch.equal(J2.view(torch.int64), J.view(torch.int64)) and torch.equal(r2, r)
    assert torch.equal(s2, s)
