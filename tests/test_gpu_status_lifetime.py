"""The status words' copy may still be queued when its context is dropped: the
pinned block it lands in is not handed out again before that, and is given back
afterwards."""
import gc
import weakref

import pytest
import torch

from helpers import scene
from warp_sph_gpt_gb300.engine import _Posted, context_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("streams", [1, 2])
def test_a_late_status_copy_reaches_no_other_pinned_tensor(streams):
    gc.collect()  # contexts of other tests
    s, P, B, D, W, grids = scene()
    ctx = context_for(P, B, D, W, tuple(grids))
    ctx.ctl[8:] = 77
    torch.cuda.synchronize()
    held = len(_Posted.dropped)
    side = torch.cuda.Stream()
    for st in [side, torch.cuda.current_stream()][2 - streams:]:
        with torch.cuda.stream(st):
            if st is side or streams == 1:
                torch.cuda._sleep(300_000_000)  # ~0.15 s of queued work, then the copy
            ctx.post_status()
    gone = weakref.ref(ctx)
    del s, P, B, D, W, grids, ctx
    gc.collect()
    assert gone() is None and len(_Posted.dropped) == held + 1
    _Posted.release_landed()
    fresh = [torch.zeros(16, dtype=torch.int32, pin_memory=True) for _ in range(4)]
    torch.cuda.synchronize()
    assert all(int(t.abs().max()) == 0 for t in fresh)
    _Posted.release_landed()
    assert not _Posted.dropped
