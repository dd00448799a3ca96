"""Tile counts on either side of the limits below which interior and last-slab
tiles share one launch (592 tiles in the predictor, 740 in the reconstruction
on 148 SMs): containers and reconstructions against the oracle, bit for bit,
plain and progressive."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# 576, 640, 704, 768 tiles, the last slabs ragged or full
SHAPES = [(121, 128, 144), (128, 121, 160), (128, 128, 170), (128, 128, 192)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", SHAPES)
def test_split(dims, dtype):
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    from prism_b200 import fields
    nx, ny, nz = dims
    data = fields.make("sinusoid", (nz, ny, nx), dtype, 3)
    d_in = torch.from_numpy(data).cuda()
    h = P.Handle()
    for prog in (False, True):
        ctx = P.Context(nx, ny, nz, np.dtype(dtype), P.REL, 1e-4, prog)
        comp = P.Compressor(ctx, h)
        cont = comp.compress_pipeline(d_in).clone()
        host = cont.cpu().numpy().tobytes()
        want, _, _ = O.compress(data, 1, 1e-4, 0 if prog else 1, force=O.intp(*comp.flags))
        assert host == want
        if not prog:
            got = comp.decompress_pipeline(cont).cpu().numpy()
            assert np.array_equal(got.view(np.uint8), O.decompress(host, data.shape, dtype, 1, 1e-4).view(np.uint8))
            continue
        pg, st = comp.progressive(cont), O.ProgressiveState()
        for target in (1e-2, 1e-4):
            got = pg.step(target).cpu().numpy()
            ref, _ = O.progressive_step(host, data.shape, dtype, 1, 1e-4, target, st)
            assert np.array_equal(got.view(np.uint8), ref.view(np.uint8))
        pg.close()
