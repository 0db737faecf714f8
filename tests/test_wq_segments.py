"""The streaming apply's plane ranges: CTAs whose ranges begin and end inside an
element, cross from one tile into the next, or hold more than 16 planes (whose
lengths then fall from one round of the SMs to the next).

Bars as in test_wq.py: FP64 within 1e-12 relative (2-norm) of the FP64 oracle,
FP32 within 2e-6.
"""
import numpy as np
import pytest

from oracle.wq_ops import WQOracle
from yeti_b200.patches import cube_patch

# (nel, p): tile planes per CTA (FP64 / FP32 on 148 SMs)
CASES = [
    ((9, 7, 11), 5),      # one plane each: every range is a part of an element
    ((31, 19, 23), 4),    # about 3 and 1.5: ranges of unequal length
    ((33, 35, 31), 2),    # about 4 and 4: ranges that cross tiles
    ((49, 37, 45), 5),    # about 17 and 9: FP64 ranges that shorten by rounds
]


@pytest.mark.gpu
@pytest.mark.parametrize("nel,p", CASES)
def test_gpu_apply_over_cut_plane_ranges(cuda_ok, nel, p):
    from yeti_b200.wq import WQElasticity
    P = cube_patch(nel, p, perturb=0.1, wrange=(0.8, 1.2), seed=3)
    clamp = {"w0": (0, 1, 2), "v1": (1,)}
    op, ref = WQElasticity(P, 1.0, 0.3, clamp), WQOracle(P, 1.0, 0.3, clamp)
    u = np.random.default_rng(5).standard_normal(op.ndof)
    k0 = ref.apply(u)
    k1 = op.eval_Ku(u)
    assert np.linalg.norm(k1 - k0) < 1e-12 * np.linalg.norm(k0)
    k2 = op.eval_Ku(u.astype(np.float32), precision="f32").astype(np.float64)
    assert np.linalg.norm(k2 - k0) < 2e-6 * np.linalg.norm(k0)


@pytest.mark.gpu
@pytest.mark.parametrize("nel,p,prec", [((6, 5, 7), 3, "f64"), ((8, 8, 8), 2, "f32"),
                                        ((31, 19, 23), 4, "f64")])
def test_gpu_applies_in_a_row_on_device_vectors(cuda_ok, nel, p, prec):
    """The output of one apply as the input of the next without a
    synchronisation, into arrays that begin off 16-byte boundaries and hold
    other values: the zeroing of an output must neither start before the
    apply that fills its input is done nor end after the additions begin."""
    import torch
    from yeti_b200 import _lib
    from yeti_b200.wq import WQElasticity
    ctx = _lib.Context(0)
    ctx.set_stream(torch.cuda.current_stream())
    op = WQElasticity(cube_patch(nel, p, perturb=0.1, seed=3), 1.0, 0.3, {"w0": (0, 1, 2)}, ctx=ctx)
    dt = torch.float64 if prec == "f64" else torch.float32
    n = op.ndof
    u = torch.from_numpy(np.random.default_rng(5).standard_normal(n)).to(dt).cuda()
    ref = [u.cpu().numpy()]
    for _ in range(4):                   # host buffers: each call synchronises
        ref.append(op.eval_Ku(ref[-1], precision=prec))
    bar = 1e-13 if prec == "f64" else 1e-5
    for off in (0, 1):
        bufs = [torch.full((n + 4,), 7.0, dtype=dt, device="cuda") for _ in range(4)]
        src = u
        for b in bufs:
            op.apply_device(src, b[off:off + n], prec)
            src = b[off:off + n]
        torch.cuda.synchronize()
        for b, r in zip(bufs, ref[1:]):
            got = b[off:off + n].cpu().numpy()
            assert np.linalg.norm(got - r) < bar * np.linalg.norm(r)
            assert float(b[off + n]) == 7.0
    ctx.set_stream(None)


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("method", ["cg", "bicgstab"])
def test_gpu_solves_from_zero_and_from_another_start(cuda_ok, method, mixed):
    """The start residual is b itself from x0 = 0 and b - K x0 otherwise, also
    when x0 holds a single tiny entry or a NaN; the residual that a mixed solve
    ends on is the one reported."""
    from yeti_b200._lib import YetiError
    from yeti_b200.wq import WQElasticity
    op = WQElasticity(cube_patch((6, 5, 7), 3, perturb=0.1, wrange=(0.8, 1.2), seed=3), 1.0, 0.3,
                      {"w0": (0, 1, 2)})
    b = op.eval_bodyforce_vector([0.1, -0.2, -1.0])
    kw = dict(rtol=1e-9, method=method, mixed=mixed, precond="fd")
    x, st = op.pcg(b, **kw)
    r = np.linalg.norm(b - op.eval_Ku(x)) / np.linalg.norm(b)
    assert r <= 1e-9 and abs(r - st["rel_residual"]) <= 1e-2 * r + 1e-13
    for x0 in (0.5 * x, np.where(np.arange(op.ndof) == op.ndof - 1, 1e-200, 0.0)):
        x2, st2 = op.pcg(b, x0=x0, **kw)
        assert st2["rel_residual"] <= 1e-9
        assert np.linalg.norm(x2 - x) < 1e-7 * np.linalg.norm(x)
    bad = np.zeros(op.ndof)
    bad[-1] = np.nan
    try:
        _, st3 = op.pcg(b, x0=bad, **kw)
        assert not st3["rel_residual"] <= 1e-9
    except YetiError as e:
        assert "EBREAKDOWN" in str(e)


@pytest.mark.gpu
@pytest.mark.parametrize("nel,p", [((5, 2, 9), 3), ((2, 2, 2), 2), ((19, 9, 4), 5), ((3, 4, 5), (2, 3, 2)),
                                   ((3, 2, 4), (2, 2, 6))])
def test_gpu_setup_of_each_precision(cuda_ok, nel, p):
    """The coefficients kept in one precision, or in both (FP32 rounded from
    FP64), give the operator, the diagonal and the load of the oracle; the free
    dofs are counted over face pairs that share a layer too."""
    from yeti_b200.wq import WQElasticity
    P = cube_patch(nel, p, perturb=0.1, wrange=(0.8, 1.2), seed=3)
    clamp = {"w0": (0, 1, 2), "w1": (1,), "u1": (1, 2)}
    ref = WQOracle(P, 1.0, 0.3, clamp)
    u = np.random.default_rng(5).standard_normal(ref.ndof)
    k0, d0, f0 = ref.apply(u), ref.diag(), ref.body_force([0.3, 0.0, -1.0])
    for have in ("f64", "f32", "both"):
        op = WQElasticity(P, 1.0, 0.3, clamp, precisions=have)
        assert op.nfree == int(op.free_mask.sum())
        if have != "f32":
            assert np.linalg.norm(op.eval_Ku(u) - k0) < 1e-12 * np.linalg.norm(k0)
            f = op.eval_bodyforce_vector([0.3, 0.0, -1.0])
            assert np.linalg.norm(f - f0) < 1e-12 * np.linalg.norm(f0)
        if have != "f64":
            k2 = op.eval_Ku(u.astype(np.float32), precision="f32").astype(np.float64)
            assert np.linalg.norm(k2 - k0) < 2e-6 * np.linalg.norm(k0)
        bar = 2e-6 if have == "f32" else 1e-12
        assert np.linalg.norm(op.diag() - d0) < bar * np.linalg.norm(d0)


@pytest.mark.gpu
def test_gpu_fp64_wait_that_runs_out_is_reported(cuda_ok):
    """FP64 from degree 4 on waits for its coefficients too: with a limit of no
    polls the apply says so, with the default limit it succeeds again."""
    from yeti_b200._lib import MEM_HOST, PREC_F64, check, lib, ptr
    from yeti_b200.wq import WQElasticity
    op = WQElasticity(cube_patch((5, 4, 6), 4, perturb=0.1, seed=3), 1.0, 0.3, {"w0": (0, 1, 2)})
    u = np.random.default_rng(5).standard_normal(op.ndof)
    ref, out = op.eval_Ku(u), np.empty_like(u)
    check(lib().yeti_wq_set_wait_limit(op.handle, 0), "yeti_wq_set_wait_limit")
    assert lib().yeti_wq_apply(op.handle, ptr(u), ptr(out), PREC_F64, MEM_HOST) == -5
    check(lib().yeti_wq_set_wait_limit(op.handle, -1), "yeti_wq_set_wait_limit")
    check(lib().yeti_wq_apply(op.handle, ptr(u), ptr(out), PREC_F64, MEM_HOST), "yeti_wq_apply")
    assert np.linalg.norm(out - ref) < 1e-13 * np.linalg.norm(ref)
