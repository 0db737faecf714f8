"""The stiffness and mass kernels' pair tiles and point chunks: element sizes
with an odd and an even number of nodes, one tile and many, points in one
chunk and in several, pair sums kept in shared memory (mass) and not, output
arrays on 8-byte boundaries.  Bit-identical to the oracle, as in
test_assembly.py and test_mass.py."""
import ctypes

import numpy as np
import pytest

import oracle
from yeti_b200.patches import cube_patch, u1_system_args
from yeti_b200.stiffmtrx_elemstorage import SYSTEM_ARG_NAMES, sys_linmat_lindef_static

# (nel, p): 8, 12, 27, 64, 125 and 210 nodes per element
CASES = [((3, 2, 2), (1, 1, 1)), ((2, 3, 2), (2, 1, 1)), ((2, 2, 3), (2, 2, 2)),
         ((2, 2, 1), (3, 3, 3)), ((2, 1, 1), (4, 4, 4)), ((1, 1, 2), (6, 5, 4))]


def _args(nel, p):
    return u1_system_args(cube_patch(nel, p, perturb=0.1, wrange=(0.8, 1.2), seed=4), E=2.1,
                          nu=0.3, rho=7.8)


def _mass_inputs(args):
    d = dict(zip(SYSTEM_ARG_NAMES, args))
    return [d[k] for k in ("activeElement", "nb_data", "COORDS3D", "IEN", "nb_elem_patch", "Nkv",
                           "Ukv", "Nijk", "weight", "Jpqr", "ELT_TYPE", "PROPS", "JPROPS", "RHO",
                           "TENSOR", "ind_dof_free", "nb_dof_free", "MCRD", "NBINT", "NNODE")]


@pytest.mark.gpu
@pytest.mark.parametrize("nel,p", CASES)
def test_gpu_stiffness_and_mass_tiles_match_oracle(cuda_ok, nel, p):
    from yeti_b200.massmtrx import build_cmassmatrix
    args = _args(nel, p)
    for got, ref in zip(sys_linmat_lindef_static(*args), oracle.sys_linmat_lindef_static(*args)):
        np.testing.assert_array_equal(got, ref)
    m = _mass_inputs(args)
    for got, ref in zip(build_cmassmatrix(*m), oracle.build_cmassmatrix(m)):
        np.testing.assert_array_equal(got, ref)


# (nel, p, Gauss points per direction): column nodes in one and in several
# groups, fewer and more functions than points, one to eight points, a layout
# whose blocks leave no room for the spacing between them
SF_CASES = [((2, 2, 2), (1, 1, 1), 2), ((2, 1, 2), (3, 1, 2), 2), ((1, 2, 2), (4, 2, 1), 3),
            ((1, 1, 2), (1, 2, 3), 4), ((1, 1, 1), (6, 5, 4), 5), ((1, 1, 1), (2, 6, 3), 6),
            ((1, 1, 1), (3, 3, 3), 7), ((1, 1, 1), (7, 2, 3), 8), ((1, 1, 1), (1, 7, 3), 7)]


@pytest.mark.gpu
@pytest.mark.parametrize("nel,p,ng", SF_CASES)
def test_gpu_sumfact_shapes_match_oracle(cuda_ok, nel, p, ng):
    args = u1_system_args(cube_patch(nel, p, perturb=0.1, wrange=(0.8, 1.2), seed=4), E=2.1, nu=0.3,
                          nbint=ng ** 3)
    k0, r0, c0, _ = oracle.sys_linmat_lindef_static(*args)
    k1, r1, c1, _ = sys_linmat_lindef_static(*args, element_kernel="sumfact")
    np.testing.assert_array_equal(r1, r0)
    np.testing.assert_array_equal(c1, c0)
    assert np.linalg.norm(k1 - k0) <= 1e-12 * np.linalg.norm(k0)   # as in test_assembly.py


@pytest.mark.gpu
def test_gpu_assembly_into_arrays_on_8_byte_boundaries(cuda_ok):
    import torch
    from yeti_b200 import _lib
    from yeti_b200.stiffmtrx_elemstorage import pack_u1_model
    args = _args((2, 2, 2), (2, 2, 2))
    pm = pack_u1_model(*args)
    n = pm.nb_data
    k = torch.full((n + 2,), -1.0, dtype=torch.float64, device="cuda")
    r = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    c, F = torch.zeros_like(r), torch.zeros(pm.nb_dof_tot, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx = _lib.default_context()
    _lib.check(_lib.lib().yeti_assemble_u1_coo_ex(
        ctx.handle, ctypes.byref(pm.struct), n, k[1:].data_ptr(), r[1:].data_ptr(),
        c[1:].data_ptr(), F.data_ptr(), _lib.MEM_DEVICE, _lib.STIFF_PAIRS), "assemble")
    ref = oracle.sys_linmat_lindef_static(*args)
    np.testing.assert_array_equal(k[1:-1].cpu().numpy(), ref[0])
    np.testing.assert_array_equal(r[1:].cpu().numpy(), ref[1])
    np.testing.assert_array_equal(c[1:].cpu().numpy(), ref[2])
    assert k[0] == -1.0 and k[-1] == -1.0


@pytest.mark.gpu
@pytest.mark.parametrize("nadj", [1, 2, 3, 4])
@pytest.mark.parametrize("nel,p", [((3, 2, 2), (2, 2, 2)), ((2, 1, 2), (3, 4, 2))])
def test_gpu_gradient_of_one_to_four_adjoints_matches_oracle(cuda_ok, nadj, nel, p):
    """The kernel for one adjoint and the one for several, points in one chunk
    and in several."""
    from yeti_b200.gradient import grad_from_system_args
    args = _args(nel, p)
    rng = np.random.default_rng(nadj)
    sol = 0.01 * rng.standard_normal((3, args[2].shape[1]))
    adj = 0.01 * rng.standard_normal((nadj, 3, args[2].shape[1]))
    for got, ref in zip(grad_from_system_args(args, sol, adj),
                        oracle.grad_lin_elast_work(args, sol, adj)):
        np.testing.assert_array_equal(got, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("keep", [1.0, 0.7, 0.3])
def test_gpu_models_with_inactive_elements(cuda_ok, keep):
    """All, most and few of the elements active: the connectivity is used as it
    comes, gathered on the device, or gathered on the host."""
    from yeti_b200._lib import YetiError
    from yeti_b200.gradient import grad_from_system_args
    args = u1_system_args(cube_patch((4, 3, 3), 2, perturb=0.1, wrange=(0.8, 1.2), seed=4),
                          rho=1.0, clamp_u0=True, load_u1=(2, 1.5))
    act = (np.random.default_rng(8).random(36) < keep).astype(np.int64)
    args[0] = act
    for got, ref in zip(sys_linmat_lindef_static(*args), oracle.sys_linmat_lindef_static(*args)):
        np.testing.assert_array_equal(got, ref)
    sol = 0.01 * np.random.default_rng(3).standard_normal((3, args[2].shape[1]))
    for got, ref in zip(grad_from_system_args(args, sol, sol[None]),
                        oracle.grad_lin_elast_work(args, sol, sol[None])):
        np.testing.assert_array_equal(got, ref)
    e = int(np.flatnonzero(act)[1])
    for wrong in (0, args[2].shape[1] + 1):
        bad = list(args)
        bad[3] = np.array(args[3])
        bad[3][27 * e + 5] = wrong
        with pytest.raises(YetiError, match=f"IEN entry {wrong} of element {e + 1} out of range"):
            sys_linmat_lindef_static(*bad)
    for got, ref in zip(sys_linmat_lindef_static(*args), oracle.sys_linmat_lindef_static(*args)):
        np.testing.assert_array_equal(got, ref)
