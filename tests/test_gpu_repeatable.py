"""Containers are the same on every call, on 1-D fields around the sizes where
threads of one round of the last shuffle block store to the same bytes (530 to
797 values), alone and in a batch.  (Against the oracle, 2-D sizes among them:
test_last_block_order.py.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_short_line_fields(dtype):
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    from prism_b200 import fields
    h = P.Handle()
    items, alone = [], []
    for nx in (513, 516, 600, 735, 900, 1002, 1023):
        d = torch.from_numpy(fields.make("grf", (1, 1, nx), dtype, nx)).cuda()
        ctx = P.Context(nx, 1, 1, np.dtype(dtype), P.REL, 1e-3, False)
        comp = P.Compressor(ctx, h)
        seen = {comp.compress_pipeline(d).cpu().numpy().tobytes() for _ in range(20)}
        assert len(seen) == 1, nx
        items.append((ctx, d))
        alone.append(seen.pop())
    b = P.Batch(items)
    for _ in range(10):
        conts, _ = b.compress()
        assert [c.cpu().numpy().tobytes() for c in conts] == alone
    b.close()
