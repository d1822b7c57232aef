"""The fused adjoint + normal equations cut into items (adjoint.cu: pieces of whole tuples, groups
of pieces): one item per run, per group and per piece give every run the same bits, equal to the
run alone, and [J r]^T [J r] of the materialised Jacobian to the rounding of the sums."""

import numpy as np
import pytest
import torch

from mikroptim_b200 import engine, workloads
from mikroptim_b200.batch import PRECISION_FP64, PRECISION_FP64_FMA, PRECISION_MIXED, ResidualLayout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP64_FMA, PRECISION_MIXED])
@pytest.mark.parametrize("variants,rings,spokes", [
    (3, 1, 1),      # 35 rays: one piece, a chunk of 35 rows
    (2, 8, 16),     # 9 pieces, an item each
    (1200, 8, 16),  # four groups
    (4200, 8, 16),  # one item per run
    (5, 7, 19),     # 133 rays per tuple: chunks that end inside a tuple
    (1, 32, 64),    # 35 pieces of 2,048 rays
])
def test_every_split_gives_the_bits_of_the_run_alone(variants, rings, spokes, precision):
    b, st, vs, x0 = workloads.sweep(variants, surfaces=6, wavelengths=7, rings=rings,
                                    spokes=spokes, precision=precision)
    lay = ResidualLayout(b.topology, st)
    gram = engine.adjoint_normal_equations_device(engine.DeviceSystemBatch(b), lay, b, vs, x0)
    for v in sorted({0, variants // 2, variants - 1}):
        one = b.take([v])
        alone = engine.adjoint_normal_equations_device(engine.DeviceSystemBatch(one), lay, one, vs,
                                                       x0[v:v + 1])
        assert torch.equal(gram[v], alone[0]), v
        if precision == PRECISION_MIXED:
            continue
        J, r, _ = engine.adjoint_jacobian_device(engine.DeviceSystemBatch(one), lay, one, vs,
                                                 x0[v:v + 1])
        X = np.concatenate([J[0].cpu().numpy(), r[0].cpu().numpy()[None]])
        want = X @ X.T
        d = np.sqrt(np.maximum(np.diagonal(want), 1e-300))
        # rows differ by the rounding of the piston (OPL of 1e5 waves: 1e-16 * 1e5 per row, the
        # residual column), sums by sqrt(rows) roundings
        err = np.abs(gram[v].cpu().numpy() - want) / (d[:, None] * d[None, :])
        assert err[:-1, :-1].max() <= 1e-12
        assert err.max() <= 1e-9


@pytest.mark.parametrize("surfaces,P", [(41, 61), (43, 64)])
def test_the_last_column_tile(surfaces, P):
    """64 variables and the residual column are 65 columns: nine column tiles, 45 pairs."""
    b, st, vs, x0 = workloads.sweep(2, surfaces=surfaces, wavelengths=2, rings=3, spokes=5,
                                    precision=PRECISION_FP64)
    assert vs.size == P
    lay = ResidualLayout(b.topology, st)
    db = engine.DeviceSystemBatch(b)
    gram = engine.adjoint_normal_equations_device(db, lay, b, vs, x0).cpu().numpy()
    J, r, _ = engine.adjoint_jacobian_device(db, lay, b, vs, x0)
    X = torch.cat([J, r[:, None]], dim=1).cpu().numpy()
    for v in range(2):
        want = X[v] @ X[v].T
        d = np.sqrt(np.maximum(np.diagonal(want), 1e-300))
        err = np.abs(gram[v] - want) / (d[:, None] * d[None, :])  # bounds as above
        assert err[:-1, :-1].max() <= 1e-12 and err.max() <= 1e-9
