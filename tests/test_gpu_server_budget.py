"""The smallest budget a server takes a field at: its container, and per slot
a workspace of codes, planes, 24 bytes a chunk, anchors and 64 KiB, plus an
eighth.  With one reconstruction more it serves the field."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(64, 48, 40), (300, 260, 40), (801, 813, 1)])
@pytest.mark.parametrize("slots", [1, 3])
def test_field_fits_its_workspace(dims, slots):
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    from prism_b200 import fields
    nx, ny, nz = dims
    data = torch.from_numpy(fields.make("sinusoid", (nz, ny, nx), np.float32, 3)).cuda()
    ctx = P.Context(nx, ny, nz, np.dtype(np.float32), P.REL, 1e-4, True)
    comp = P.Compressor(ctx)
    cont = comp.compress_pipeline(data).clone()
    g = O.geometry(nx, ny, nz, 4)
    w = 4 * int(P.lib().prism_code_buffer_len(nx, ny, nz)) + int(g.aligned_size) + 64 + 24 * int(g.chunks) \
        + 16 * int(g.anchors) + 65536
    least = slots * (w + w // 8) + cont.numel()
    srv = P.Server(least - 1, slots=slots)
    with pytest.raises(P.PrismError):
        srv.add_field(ctx, cont)
    srv.close()
    srv = P.Server(least + 4 * nx * ny * nz, slots=slots)
    fid = srv.add_field(ctx, cont)
    assert srv.stats()["bytes_reserved"] == least - cont.numel()
    out = torch.empty_like(data)
    srv.wait(srv.submit(fid, 1e-2, out))
    prog = comp.progressive(cont)
    assert torch.equal(prog.step(1e-2), out)
    prog.close()
    srv.close()
