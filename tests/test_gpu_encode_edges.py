"""Chunks at the encoder's size limits in the pipeline, which codes its plane
buffer in place: chunks whose bytes and first bitmap alone reach the chunk
size, chunks that only the last bitmaps decide (a rejected one must stay as it
is in the buffer), and sizes one below, at and one above the chunk's."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

CHUNK = 16384
BOUNDS = (2.0, 1.5, 1.2, 1.0, 0.9, 0.4)


def chunk_kinds(planes, g):
    """Per chunk of the plane buffer: how the coder decides, and the coded
    size minus the chunk's size where the last bitmaps decide."""
    kinds, over, at = set(), set(), 0
    for l in (3, 2, 1, 0):
        st = int(g.hastride[l])
        for p in range(32):
            for o in range(0, st, CHUNK):
                c = planes[at + p * st + o:at + p * st + min(o + CHUNK, st)]
                nz, bm = int((c != 0).sum()), np.zeros(2048, np.uint8)
                packed = np.packbits(c != 0, bitorder="little")
                bm[:packed.size] = packed
                kept = []
                for _ in range(3):
                    f = bm != np.concatenate([[0], bm[:-1]])
                    kept.append(int(f.sum()))
                    bm = np.packbits(f, bitorder="little")
                if nz == 0:
                    kinds.add("zero")
                elif nz + kept[0] + 6 >= c.size:
                    kinds.add("raw")
                elif nz + kept[0] + 6 + 288 < c.size:
                    kinds.add("coded early")
                else:
                    d = nz + sum(kept) + 6 - c.size
                    over.add(d)
                    kinds.add("coded late" if d < 0 else "rejected late")
        at += 32 * st
    return kinds, over


def test_chunks_at_the_size_limits():
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    shape = nz, ny, nx = 64, 64, 128
    data = np.random.default_rng(1).standard_normal(shape).astype(np.float32)
    d_in, g, h = torch.from_numpy(data).cuda(), O.geometry(nx, ny, nz, 4), P.Handle()
    kinds, over = set(), set()
    for prog in (False, True):
        for bound in BOUNDS:
            comp = P.Compressor(P.Context(nx, ny, nz, np.dtype(np.float32), P.ABS, bound, prog), h)
            got = comp.compress_pipeline(d_in).cpu().numpy().tobytes()
            bt = 0 if prog else 1
            want, _, _ = O.compress(data, 0, bound, bt, force=O.intp(*comp.flags))
            assert got == want, (prog, bound)
            _, qc, scratch = O.predict(data, bound, *comp.flags, 0.0)
            k, o = chunk_kinds(O.bitshuffle(qc, g, bt, scratch)[:int(g.aligned_size)], g)
            kinds |= k
            over |= o
    assert kinds == {"zero", "raw", "coded early", "coded late", "rejected late"}
    assert {-1, 0, 1} <= over
    h.close()
