"""The 16-byte pieces in which the fast-diagonalisation passes stage a row.

A row of m free values is staged in pieces of 16 bytes up to a whole matrix
step (m rounded up to a multiple of 4), so that in FP64 the last piece of m = 4 j
+ 1 values lies beyond the row: it must read nothing.  Rows take this path when
they begin on 16 bytes, as with an even number of functions along u and no
component clamped at u0; clamped at u1, the free size is odd.

GPU tolerances as in test_fd_tiles.py (the same products), against its dense
products after one step of refinement: scipy's eigenvalues are good to a
rounding of the largest, which on 66x63x2 elements is 2e-12 of the result.
"""
import os
import subprocess

import numpy as np
import pytest

from oracle.wq_ops import WQOracle
from test_fd_tiles import _dense
from yeti_b200 import build
from yeti_b200.patches import cube_patch

PIECES = r"""
#include <cstdio>
#include "fd_stage.cuh"
int main() {
    for (int vec : {2, 4})
        for (int m = 1; m <= 512; m++)
            for (int k = 0; k < yeti::fd_m4(m); k += vec)
                std::printf("%d %d %d %d\n", vec, m, k, yeti::fd_piece(m, k, vec));
}
"""


def test_pieces_cover_a_row_and_nothing_else(tmp_path):
    src, exe = tmp_path / "pieces.cpp", tmp_path / "pieces"
    src.write_text(PIECES)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, "-I", cuda, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    vec, m, k, n = np.loadtxt(out.splitlines(), dtype=np.int64).T
    assert n.min() >= 0 and (n <= vec).all()
    np.testing.assert_array_equal(n, np.clip(m - k, 0, vec))
    assert (k[n > 0] + n[n > 0] <= m[n > 0]).all()
    for v in (2, 4):
        covered = np.bincount(m[vec == v], weights=n[vec == v], minlength=513)
        np.testing.assert_array_equal(covered, np.arange(513))


ALL, ONE = {"u1": (0, 1, 2)}, {"u1": (0,), "w0": (1, 2)}
CASES = [((nu, 4, 3), p, clamp)                     # planes; free along u: m of
         for nu, p in ((9, 3), (11, 3), (14, 4))    # 11, 13, 17 (12, 14, 18 where
         for clamp in (ALL, ONE)] + [               # the component is not clamped)
    ((63, 3, 2), 3, ALL),                           # 65 6 5: planes
    ((64, 64, 2), 2, ALL),                          # 65 66 4: lines in FP64
    ((66, 63, 2), 2, ONE),                          # 67/68 65 3/4: lines in FP64
    ((64, 64, 2), 4, ONE),                          # 67/68 68 5/6: lines in FP64
]


def _solved(P, clamp, r):
    """P^-1 r of the separable operator, from its eigenvectors and corrected
    by its residual in extended precision."""
    ref = WQOracle(P, 1.0, 0.3, clamp)
    z = _dense(P, clamp, r)
    res = r.astype(np.longdouble).reshape(3, *ref.n[::-1])
    x = z.astype(np.longdouble).reshape(res.shape)
    for c in range(3):
        box = ref.fd_box(c)
        (Ku, Mu), (Kv, Mv), (Kw, Mw) = [[A.astype(np.longdouble) for A in ref.fd_1d(d, lo, hi)]
                                        for d, (lo, hi) in enumerate(box)]
        sl = tuple(slice(lo, hi) for lo, hi in box[::-1])
        for A, B, C in ((Kw, Mv, Mu), (Mw, Kv, Mu), (Mw, Mv, Ku)):
            y = np.tensordot(A, x[c][sl], (1, 0))
            y = np.moveaxis(np.tensordot(B, y, (1, 1)), 0, 1)
            res[c][sl] -= np.moveaxis(np.tensordot(C, y, (1, 2)), 0, 2)
    return z + _dense(P, clamp, res.astype(np.float64).ravel())


@pytest.mark.gpu
@pytest.mark.parametrize("nel,p,clamp", CASES)
def test_gpu_rows_clamped_at_their_end(cuda_ok, nel, p, clamp):
    """... beside intermediates whose memory holds NaN off the free boxes,
    left there by an operator whose boxes end one plane later along u."""
    from yeti_b200._lib import PREC_F32, PREC_F64, Context
    from yeti_b200.wq import WQElasticity
    P = cube_patch(nel, p, perturb=0.1, wrange=(0.9, 1.1), seed=6)
    ctx = Context(0)
    before = WQElasticity(P, 1.0, 0.3, {"w1": (0, 1, 2)}, ctx=ctx)
    for prec, dtype in ((PREC_F64, np.float64), (PREC_F32, np.float32)):
        assert np.isnan(before.fd_apply(np.full(before.ndof, np.nan, dtype), "fd_unit", prec)).any()
    before.close()
    op = WQElasticity(P, 1.0, 0.3, clamp, ctx=ctx)
    r = np.random.default_rng(2).standard_normal(op.ndof) * op.free_mask
    z0 = _solved(P, clamp, r)
    z = op.fd_apply(r, "fd_unit", PREC_F64)
    assert np.linalg.norm(z - z0) < 1e-12 * np.linalg.norm(z0)
    z32 = op.fd_apply(r.astype(np.float32), "fd_unit", PREC_F32).astype(np.float64)
    assert np.linalg.norm(z32 - z0) < 2e-5 * np.linalg.norm(z0)
    op.close()
    ctx.close()
