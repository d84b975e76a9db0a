"""The status words' copy may still be queued when its context is dropped: the
pinned block it lands in is not handed out again before that."""
import gc
import weakref

import pytest
import torch

from helpers import scene
from warp_sph_gpt_gb300.engine import context_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("posts", [1, 3])
def test_a_late_status_copy_reaches_no_other_pinned_tensor(posts):
    s, P, B, D, W, grids = scene()
    ctx = context_for(P, B, D, W, tuple(grids))
    ctx.ctl[8:] = 77
    torch.cuda.synchronize()
    torch.cuda._sleep(300_000_000)  # ~0.15 s of queued work, then the copies
    for _ in range(posts):
        ctx.post_status()
    gone = weakref.ref(ctx)
    del s, P, B, D, W, grids, ctx
    gc.collect()
    assert gone() is None
    fresh = [torch.zeros(16, dtype=torch.int32, pin_memory=True) for _ in range(4)]
    torch.cuda.synchronize()
    assert all(int(t.abs().max()) == 0 for t in fresh)
