"""The FP64 cycle's smallest levels in one block (csrc/cycle_tail.cu) against
the oracle's V-cycle on the exported hierarchy."""
import numpy as np
import pytest

import cfdx_dev_b200 as cg
from tests import cases

pytestmark = pytest.mark.gpu


def _pressure_system(ctx, m):
    mesh = cg.Mesh(ctx, m)
    U, rAU, aP, p, fixed, value = cases.simple_fields(m, mesh.geometry()["cell_centres"])
    A, b, _, _ = cg.assemble_pressure_correction(mesh, U, rAU, p, 1.0, fixed, value)
    return A, b


@pytest.mark.parametrize("kind,options", [
    ("tet1", {}),                        # six rows: one level, the dense LU
    ("tet3", {}),                        # 162 rows: the whole cycle in the tail
    ("tet8", {}),                        # 3,072 rows: the tail starts below the fine level
    ("tet14", {}),                       # 16,464 rows
    ("layer", {}),                       # ends in the <= 16-row LU
    ("tet3", dict(max_levels=1)),        # one level, 24 sweeps
    ("tet6", dict(max_levels=3)),        # a coarsest level of a few hundred rows, swept
    ("tet6", dict(pre_sweeps=0, post_sweeps=1)),
    ("tet6", dict(pre_sweeps=2, post_sweeps=3, coarse_pre_sweeps=0, coarse_post_sweeps=1)),
    ("tet6", dict(narrow_columns=0)),
])
def test_tail_matches_the_oracle_cycle(ctx, oracle, kind, options):
    """FP64 sums in another order: 1e-13, as the cycle's default row order is held to elsewhere."""
    m = cg.boundary_layer_case(10, 14, 6) if kind == "layer" else cases.simple_mesh(int(kind[3:]))
    A, b = _pressure_system(ctx, m)
    fast = cg.NativeBoomerAMGPreconditioner(ctx, **options)
    exact = cg.NativeBoomerAMGPreconditioner(ctx, reference_order=1, **options)
    assert fast.setup(A) and exact.setup(A)
    for seed in (1, 2):
        r = np.random.default_rng(seed).standard_normal(A.n)
        z, z_ref = fast.apply(r), exact.apply(r)
        assert np.linalg.norm(z - z_ref) <= 1e-13 * np.linalg.norm(z_ref)
        assert np.array_equal(z, fast.apply(r))          # deterministic
    if not options:
        H = oracle.Hierarchy([exact.export_level(l) for l in range(len(exact.hierarchy_level_sizes()))], exact.omega)
        assert np.array_equal(z_ref, H.apply(r))         # the yardstick is the reference's cycle
    # refreshed values and damping reach the tail
    ro, co, va = A.to_csr()
    B = cg.SparseMatrix.from_csr(ctx, ro, co, 3.0 * va)
    assert fast.update_values(B) and exact.update_values(B)
    z, z_ref = fast.apply(r), exact.apply(r)
    assert np.linalg.norm(z - z_ref) <= 1e-13 * np.linalg.norm(z_ref)


def test_tail_reports_non_finite_input(ctx):
    A, b = _pressure_system(ctx, cases.simple_mesh(3))
    amg = cg.NativeBoomerAMGPreconditioner(ctx)
    assert amg.setup(A)
    b[5] = np.inf
    with pytest.raises(cg.CfdxgError):
        amg.apply(b)
