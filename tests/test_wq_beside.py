"""Small applies start beside the zeroing of their output (a programmatic
dependent launch): what the caller has on the stream before and after them
keeps its place, also when an apply gives up a wait and returns early.

Tolerances of a chain of four applies: each is within 1e-12 (FP64) or 2e-6
(FP32) of the operator, the bars of the other tests; four of them, 4e-12 and
8e-6.
"""
import numpy as np
import pytest

from yeti_b200.patches import cube_patch

CASES = [((6, 5, 7), 3, "f32"), ((5, 4, 6), 4, "f64"), ((8, 8, 8), 2, "f64")]


def _setup(nel, p, prec):
    import torch
    from yeti_b200._lib import Context
    from yeti_b200.wq import WQElasticity
    ctx, stream = Context(0), torch.cuda.Stream()
    ctx.set_stream(stream)
    op = WQElasticity(cube_patch(nel, p, perturb=0.1, seed=3), 1.0, 0.3, {"w0": (0, 1, 2)}, ctx=ctx)
    u = np.random.default_rng(5).standard_normal(op.ndof)
    dt = torch.float32 if prec == "f32" else torch.float64
    return ctx, stream, op, u, torch.tensor(u, dtype=dt, device="cuda")


@pytest.mark.gpu
@pytest.mark.parametrize("nel,p,prec", CASES)
def test_gpu_kernels_of_the_caller_between_applies(cuda_ok, nel, p, prec):
    import torch
    ctx, stream, op, u, x = _setup(nel, p, prec)
    ref = u.copy()
    for s in (0.5, 2.0, 1.0, 4.0):
        ref = op.eval_Ku(ref) * s
    y, z = torch.empty_like(x), torch.empty_like(x)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for _ in range(5):                   # nothing waits on the host
            op.apply_device(x, y, prec)
            y.mul_(0.5)                      # between two applies
            op.apply_device(y, z, prec)
            z.mul_(2.0)
            y.fill_(float("nan"))            # read by the apply before, written by the next
            op.apply_device(z, y, prec)
            op.apply_device(y, z, prec)      # no kernel between
            z.mul_(4.0)
        got = z.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - ref) < (8e-6 if prec == "f32" else 4e-12) * np.linalg.norm(ref)
    op.close()
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nel,p,prec", CASES[:2])
def test_gpu_what_follows_an_apply_that_gave_up(cuda_ok, nel, p, prec):
    """Degrees whose applies wait for coefficient copies: with a limit of no
    polls every CTA returns early, and a kernel that follows still finds the
    zeroing done."""
    import torch
    from yeti_b200._lib import check, lib
    ctx, stream, op, u, x = _setup(nel, p, prec)
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    check(lib().yeti_wq_set_wait_limit(op.handle, 0), "yeti_wq_set_wait_limit")
    kept = []
    with torch.cuda.stream(stream):
        for k in range(50):
            op.apply_device(x, y, prec)
            y.fill_(k + 1)
            kept.append((y == k + 1).all())
    stream.synchronize()
    assert all(bool(k) for k in kept)
    assert bool((y == 50).all())
    op.close()
    ctx.close()
