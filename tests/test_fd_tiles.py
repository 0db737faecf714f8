"""The fast-diagonalisation passes at the edges of their tilings: free sizes
just below, at and above the rows and lines of a unit (4, 8, 16) and of a whole
matrix step, rows that begin on 16 bytes and rows that do not, planes that fit
one CTA and planes that do not, and components whose boxes differ.

FP64 within 1e-12 relative (2-norm) of the same eigenvectors applied by dense
products: the sums have at most 140 terms of either sign, three times over, so
the bar is some hundred roundings.  FP32 within 2e-5, as for any FP32 chain of
six such products of operands rounded to FP32.
"""
import numpy as np
import pytest
import scipy.linalg

from oracle.wq_ops import WQOracle
from yeti_b200.patches import cube_patch

# (nel, p, clamp): free functions per direction
CASES = [
    ((2, 2, 2), 2, {"w0": (0, 1, 2)}),                       # 4 4 3
    ((5, 6, 7), 2, {"w0": (0, 1, 2)}),                       # 7 8 8
    ((6, 7, 13), 2, {"u0": (0, 1, 2), "v1": (1,)}),          # 7 9/8 15
    ((13, 14, 15), 3, {"w0": (0, 1, 2), "w1": (0, 1, 2)}),   # 16 17 16
    ((61, 3, 30), 3, {"u1": (0, 1, 2)}),                     # 63 6 33
    ((4, 60, 5), 4, {"v0": (0, 1, 2)}),                      # 8 63 9
    ((136, 5, 3), 4, {"w0": (0, 1, 2)}),                     # 140 9 6: lines pass
    ((3, 4, 130), 3, {"w1": (0, 1, 2)}),                     # 6 7 132
]


def _dense(P, clamp, r):
    """U (a / Lambda) U^T r per component, from scipy's eigenvectors."""
    ref = WQOracle(P, 1.0, 0.3, clamp)
    n = ref.n
    r = r.reshape(3, n[2], n[1], n[0])
    out = np.zeros_like(r)
    for c in range(3):
        box = ref.fd_box(c)
        lam, U = [], []
        for d, (lo, hi) in enumerate(box):
            K, M = ref.fd_1d(d, lo, hi)
            w, v = scipy.linalg.eigh(K, M)
            lam.append(w)
            U.append(v)
        sl = tuple(slice(lo, hi) for lo, hi in box[::-1])
        x = np.einsum("wvu,ua->wva", r[c][sl], U[0], optimize=True)
        x = np.einsum("wva,vb->wba", x, U[1], optimize=True)
        x = np.einsum("wba,wc->cba", x, U[2], optimize=True)
        x = x / (lam[0][None, None, :] + lam[1][None, :, None] + lam[2][:, None, None])
        x = np.einsum("cba,wc->wba", x, U[2], optimize=True)
        x = np.einsum("wba,vb->wva", x, U[1], optimize=True)
        out[c][sl] = np.einsum("wva,ua->wvu", x, U[0], optimize=True)
    return out.ravel()


@pytest.mark.gpu
@pytest.mark.parametrize("nel,p,clamp", CASES)
def test_gpu_fd_passes_match_dense_products(cuda_ok, nel, p, clamp):
    from yeti_b200._lib import PREC_F32, PREC_F64
    from yeti_b200.wq import WQElasticity
    full = {k: (0, 1, 2) if k != "v1" else v for k, v in clamp.items()}
    P = cube_patch(nel, p, perturb=0.1, wrange=(0.9, 1.1), seed=6)
    op = WQElasticity(P, 1.0, 0.3, full)
    r = np.random.default_rng(2).standard_normal(op.ndof) * op.free_mask
    z0 = _dense(P, full, r)
    z = op.fd_apply(r, "fd_unit", PREC_F64)
    assert np.linalg.norm(z - z0) < 1e-12 * np.linalg.norm(z0)
    z32 = op.fd_apply(r.astype(np.float32), "fd_unit", PREC_F32).astype(np.float64)
    assert np.linalg.norm(z32 - z0) < 2e-5 * np.linalg.norm(z0)
