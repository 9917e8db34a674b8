"""Dense coarse inverse of the FP32 cycle (csrc/dense.cu): a system of at most
coarse_dense_limit rows is one level, whose cycle is the inverse itself."""
import numpy as np
import pytest

import cfdx_dev_b200 as cg

pytestmark = pytest.mark.gpu


def _system(n, seed, shift, skew=0.0):
    """Symmetric M-matrix with random couplings (about eight per row) plus shift, optionally skewed."""
    rng = np.random.default_rng(seed)
    a = np.zeros((n, n))
    for _ in range(4):
        i = rng.permutation(n)
        w = rng.uniform(0.1, 1.0, n)
        a[np.arange(n), i] -= w
        a[i, np.arange(n)] -= w
    np.fill_diagonal(a, 0.0)
    np.fill_diagonal(a, -a.sum(1) + shift)
    if skew and n > 1:
        a[0, 1] -= skew
    rows, cols = np.nonzero(a)
    ro = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int64)
    return a, ro, cols.astype(np.int64), a[rows, cols]


@pytest.mark.parametrize("dense_fp64", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 130, 1000, 1537])
def test_dense_inverse_of_an_spd_level(ctx, n, dense_fp64):
    """One row, remainders and multiples of the 64-wide blocks, odd row lengths.
    The cycle rounds r and z to FP32 (2^-24 each) and reads the inverse as FP32
    or FP64; the systems' condition is below 40."""
    a, ro, co, va = _system(n, n, 1.0)
    A = cg.SparseMatrix.from_csr(ctx, ro, co, va)
    amg = cg.NativeBoomerAMGPreconditioner(ctx, precision="fp32_vcycle", dense_fp64=dense_fp64)
    assert amg.setup(A), amg.last_error()
    assert len(amg.hierarchy_level_sizes()) >= 1
    r = np.random.default_rng(7).standard_normal(n)
    z = np.linalg.solve(a, r)
    assert np.linalg.norm(amg.apply(r) - z) <= 40 * 2.0 ** -23 * np.linalg.norm(z)
    # a refresh on new values re-forms it
    B = cg.SparseMatrix.from_csr(ctx, ro, co, 2.0 * va)
    assert amg.update_values(B)
    assert np.linalg.norm(amg.apply(r) - 0.5 * z) <= 40 * 2.0 ** -23 * np.linalg.norm(0.5 * z)


def test_nonsymmetric_level_pays_for_lu_alone(ctx):
    """A refresh of a level that is not symmetric launches none of the two
    kernels per 64 columns of the symmetric route, and keeps two n x n FP64
    arrays beside the FP32 inverse and the solver's own memory (315 MB here);
    a third would be 128 MB more."""
    import torch
    n = 4000
    i = np.arange(n)
    a = np.zeros((n, n))
    a[i, i] = 3.0
    a[i[1:], i[:-1]] = a[i[:-1], i[1:]] = -1.0
    launches = {}
    for skew in (0.0, 0.3):
        a[0, 1] = -1.0 - skew
        rows, cols = np.nonzero(a)
        ro = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int64)
        A = cg.SparseMatrix.from_csr(ctx, ro, cols.astype(np.int64), a[rows, cols])
        r = np.random.default_rng(7).standard_normal(n)
        z = np.linalg.solve(a, r)
        for _ in range(2):   # the first one loads the solver's own code
            free = torch.cuda.mem_get_info()[0]
            amg = cg.NativeBoomerAMGPreconditioner(ctx, precision="fp32_vcycle")
            assert amg.setup(A), amg.last_error()
            used = free - torch.cuda.mem_get_info()[0]
            before = ctx.kernel_launches
            assert amg.update_values(A)
            launches[skew] = ctx.kernel_launches - before
            assert np.linalg.norm(amg.apply(r) - z) <= 40 * 2.0 ** -23 * np.linalg.norm(z)
            del amg
    assert launches[0.3] < launches[0.0] - 100
    assert used <= (2 * 8 + 4) * n * n + 380e6


def test_dense_inverse_of_a_nonsymmetric_level(ctx):
    """Not symmetric: the LU route, with the same result."""
    a, ro, co, va = _system(200, 3, 1.0, skew=0.3)
    amg = cg.NativeBoomerAMGPreconditioner(ctx, precision="fp32_vcycle")
    assert amg.setup(cg.SparseMatrix.from_csr(ctx, ro, co, va)), amg.last_error()
    r = np.random.default_rng(7).standard_normal(200)
    z = np.linalg.solve(a, r)
    assert np.linalg.norm(amg.apply(r) - z) <= 40 * 2.0 ** -23 * np.linalg.norm(z)
