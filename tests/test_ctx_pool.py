"""The context's pool of freed blocks: calls of several sizes reuse it, also
from one stream to the next and beside an HBM budget."""
import numpy as np
import pytest

import oracle
from yeti_b200.patches import cube_patch, u1_system_args
from yeti_b200.stiffmtrx_elemstorage import sys_linmat_lindef_static


def _args(nel, seed):
    return u1_system_args(cube_patch(nel, 2, perturb=0.1, wrange=(0.8, 1.2), seed=seed),
                          clamp_u0=True, load_u1=(3, -1.0))


@pytest.mark.gpu
def test_calls_on_changing_streams_reuse_freed_blocks(cuda_ok):
    import torch
    from yeti_b200._lib import Context
    ctx = Context(0)
    streams = [None, torch.cuda.Stream(), torch.cuda.Stream()]
    models = [_args(nel, k) for k, nel in enumerate([(3, 2, 2), (5, 4, 3), (2, 2, 2), (5, 4, 3)])]
    refs = [oracle.sys_linmat_lindef_static(*a) for a in models]
    for rnd in range(3):
        for k, (a, ref) in enumerate(zip(models, refs)):
            ctx.set_stream(streams[(k + rnd) % 3])
            for got, want in zip(sys_linmat_lindef_static(*a, ctx=ctx), ref):
                np.testing.assert_array_equal(got, want)
            assert ctx.bytes_in_use() == 0
    ctx.close()


@pytest.mark.gpu
def test_a_kept_block_does_not_count_against_the_budget(cuda_ok):
    from yeti_b200._lib import Context, YetiError
    big, small = _args((6, 5, 4), 1), _args((3, 2, 2), 2)
    need = int(big[1]) * 16          # the COO arrays of the larger model
    ctx = Context(0, hbm_budget_bytes=need + (1 << 20))
    want = oracle.sys_linmat_lindef_static(*big)[0]
    for _ in range(3):               # the small call's blocks give way each time
        sys_linmat_lindef_static(*small, ctx=ctx)
        np.testing.assert_array_equal(sys_linmat_lindef_static(*big, ctx=ctx)[0], want)
    ctx.close()
    ctx = Context(0, hbm_budget_bytes=need // 2)
    sys_linmat_lindef_static(*small, ctx=ctx)
    with pytest.raises(YetiError, match="ENOMEM"):
        sys_linmat_lindef_static(*big, ctx=ctx)
    sys_linmat_lindef_static(*small, ctx=ctx)
    ctx.close()


@pytest.mark.gpu
def test_operators_rebuilt_over_freed_ones(cuda_ok):
    """A design loop's pattern: operators set up, applied on one stream and
    destroyed after the context has moved to another."""
    import torch
    from yeti_b200._lib import Context
    from yeti_b200.wq import WQElasticity
    ctx = Context(0)
    out = []
    for k in range(4):
        ctx.set_stream(torch.cuda.Stream())
        op = WQElasticity(cube_patch((6, 5, 7), 3, perturb=0.1, seed=k % 2), 1.0, 0.3,
                          {"w0": (0, 1, 2)}, ctx=ctx)
        u = np.random.default_rng(1).standard_normal(op.ndof)
        out.append(op.eval_Ku(u))
        ctx.set_stream(None)
        op.close()
    for a, b in ((0, 2), (1, 3)):
        assert np.linalg.norm(out[a] - out[b]) < 1e-13 * np.linalg.norm(out[a])
    ctx.close()


@pytest.mark.gpu
def test_a_full_pool_keeps_the_blocks_freed_last(cuda_ok):
    """Operators of many sizes fill the pool; the calls after them find their
    blocks in it all the same, and it stays within its 512 MiB."""
    import torch
    from yeti_b200._lib import Context
    from yeti_b200.wq import WQElasticity
    ctx = Context(0)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def build(nel):
        op = WQElasticity(cube_patch(nel, 3, perturb=0.1, seed=1), 1.0, 0.3, {"w0": (0, 1, 2)}, ctx=ctx)
        out = op.eval_Ku(np.ones(op.ndof))
        op.close()
        return out
    build((2, 2, 2))
    start = free()
    for n in (16, 20, 24, 26, 28, 30):
        build((n, n, n))
    assert start - free() <= (512 + 64) << 20      # and cudaMalloc's own rounding
    ref, kept = build((32, 24, 28)), free()
    for _ in range(3):
        again = build((32, 24, 28))
        assert np.linalg.norm(again - ref) < 1e-13 * np.linalg.norm(ref)
        assert abs(free() - kept) <= 8 << 20
    ctx.close()
    assert start - free() <= 64 << 20
