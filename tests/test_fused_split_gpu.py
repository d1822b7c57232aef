"""The fused adjoint + normal equations cut into items (adjoint.cu: pieces of whole tuples, groups
of pieces): one item per run, per group and per piece give every run the same bits, equal to the
run alone, and [J r]^T [J r] of the materialised Jacobian to the rounding of the sums."""

import dataclasses

import numpy as np
import pytest
import torch

from mikroptim_b200 import engine, workloads
from mikroptim_b200.batch import PRECISION_FP64, PRECISION_FP64_FMA, PRECISION_MIXED, ResidualLayout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP64_FMA, PRECISION_MIXED])
@pytest.mark.parametrize("variants,rings,spokes", [
    (3, 1, 1),      # 35 rays: one piece, a chunk of 35 rows on a block of 128
    (2, 8, 16),     # 9 pieces, an item each
    (1200, 8, 16),  # one item per run (FP64), four groups (MIXED)
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


# 4,480 rays are 9 pieces on blocks of 256 rays, 2,240 are 9 on blocks of 128. One item per run from
# eight runs per block of the GPU on, one per group from two: 148 (FP64) and 296 (MIXED) blocks of
# 256, 444 and 592 of 128, so 1,000 and 1,500 runs are cut into groups in every precision.
@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP64_FMA, PRECISION_MIXED])
@pytest.mark.parametrize("variants,rings,spokes,items", [
    (2, 8, 16, 9), (1000, 8, 16, 4), (4200, 8, 16, 1),
    (3, 4, 16, 9), (1500, 4, 16, 4), (5000, 4, 16, 1),
    (3, 5, 11, 5),   # 55 rays per tuple: pieces of 495, the last two of 220
    (5, 1, 8, 1),    # 280 rays, one piece
    (2, 1, 4, 1),    # 140 rays, a chunk and a part
])
def test_items_per_run_and_their_sums(monkeypatch, variants, rings, spokes, items, precision):
    """The split that the batch size asks for is the one taken (the runs' item counters, after the
    records and the queue counter in the workspace), and its sums are the run's alone."""
    b, st, vs, x0 = workloads.sweep(variants, surfaces=6, wavelengths=7, rings=rings,
                                    spokes=spokes, precision=precision)
    lay = ResidualLayout(b.topology, st)
    db = engine.DeviceSystemBatch(b)
    made, empty = [], torch.empty

    def keep(*args, **kwargs):
        made.append(empty(*args, **kwargs))
        return made[-1]
    monkeypatch.setattr(torch, "empty", keep)
    gram = engine.adjoint_normal_equations_device(db, lay, b, vs, x0)
    monkeypatch.undo()
    torch.cuda.synchronize()
    ws = next(t for t in made if t.dtype == torch.uint8)
    at = -(-8 * variants * db.stride // 256) * 256 + 256
    done = ws[at:at + 4 * variants].view(torch.int32)
    assert (done == (items if items > 1 else 0)).all()
    for v in sorted({0, variants // 2, variants - 1}):
        one = b.take([v])
        alone = engine.adjoint_normal_equations_device(engine.DeviceSystemBatch(one), lay, one, vs,
                                                       x0[v:v + 1])
        assert torch.equal(gram[v], alone[0]), v
        J, r, _ = engine.adjoint_jacobian_device(
            engine.DeviceSystemBatch(one),
            ResidualLayout(b.topology, dataclasses.replace(st, precision=PRECISION_FP64)), one, vs,
            x0[v:v + 1])
        X = np.concatenate([J[0].cpu().numpy(), r[0].cpu().numpy()[None]])
        want = X @ X.T
        d = np.sqrt(np.maximum(np.diagonal(want), 1e-300))
        err = np.abs(gram[v].cpu().numpy() - want) / (d[:, None] * d[None, :])
        if precision == PRECISION_MIXED:  # FP32 rows: every entry within 2e-3
            assert err.max() <= 2e-3
        else:  # bounds as above
            assert err[:-1, :-1].max() <= 1e-12 and err.max() <= 1e-9
