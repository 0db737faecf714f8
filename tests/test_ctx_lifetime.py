"""Operators outlive the handle of their context, in any order of destruction
(a cycle that holds both is collected in no order that could be relied on)."""
import gc

import numpy as np
import pytest

from yeti_b200.patches import cube_patch


def _op(ctx):
    from yeti_b200.wq import WQElasticity
    return WQElasticity(cube_patch((6, 5, 7), 3, perturb=0.1, seed=1), 1.0, 0.3, {"w0": (0, 1, 2)}, ctx=ctx)


@pytest.mark.gpu
def test_operators_of_a_closed_context(cuda_ok):
    from yeti_b200._lib import Context
    ctx = Context(0)
    ops = [_op(ctx), _op(ctx)]
    u = np.random.default_rng(1).standard_normal(ops[0].ndof)
    ref = ops[0].eval_Ku(u)
    x = ops[0].fd_apply(u * ops[0].free_mask, "fd")
    ctx.close()
    for op in ops:
        got = op.eval_Ku(u)
        assert np.linalg.norm(got - ref) < 1e-13 * np.linalg.norm(ref)
        z = op.fd_apply(u * op.free_mask, "fd")
        assert np.linalg.norm(z - x) < 1e-12 * np.linalg.norm(x)
        op.close()


@pytest.mark.gpu
def test_context_and_operator_collected_together(cuda_ok):
    import torch
    from yeti_b200._lib import Context
    _op(None).close()                     # the default context's pool is filled

    def cycle(context_first):
        ctx = Context(0)
        op = _op(ctx)
        op.eval_Ku(np.ones(op.ndof))
        objs = [ctx, op] if context_first else [op, ctx]
        for a, b in zip(objs, objs[::-1]):
            a.other = b
    for first in (True, False):
        cycle(first)
        gc.collect()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for k in range(6):
        cycle(k % 2 == 0)
        gc.collect()
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 8 << 20
