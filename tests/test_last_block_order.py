"""Fields where threads of one round of the last shuffle block store to the
same bytes (zero words past the end of a plane spill onto the next one): 1-D
fields of about 513 to 800 values and small 2-D ones.  The reference's outcome
there is a race between its warps; the library and the oracle store byte j of
every word of the round before byte j + 1."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import prism_b200 as P

DIMS = [(n, 1, 1) for n in (513, 529, 530, 535, 542, 600, 661, 735, 794, 797, 798, 900, 1023)] + \
       [(17, 31, 1), (17, 35, 1), (20, 27, 1), (33, 16, 1), (33, 17, 1), (40, 15, 1)]
SAME = [(513, 1, 1), (529, 1, 1), (798, 1, 1), (900, 1, 1), (1023, 1, 1)]  # no byte stored twice in a round


def planes_of(dims, by_words):
    """Planes and codes of a code array with every plane's bit set."""
    g = O.geometry(*dims, 4)
    nx, ny, nz = dims
    n, na = int(g.n), int(g.anchors)
    c0 = n - ((nx + 1) // 2) * ((ny + 1) // 2) * ((nz + 1) // 2)
    qc = np.zeros(n + na + 2 * 16384 + 64, dtype=np.int32)
    qc[na:int(g.lm_prefix[0]) + c0] = -0x55555555  # negabinary 0xffffffff
    order = C.c_int.in_dll(O.lib(), "or_last_block_by_words")
    order.value = by_words
    try:
        planes = O.bitshuffle(qc, g, 0, np.zeros(int(g.aligned_size) + (1 << 20), dtype=np.uint8))
    finally:
        order.value = 0
    back = O.inverse_bitshuffle(planes, g, 0)
    level0 = slice(int(g.lm_prefix[0]), int(g.lm_prefix[0]) + c0)
    return planes, int(np.count_nonzero(qc[level0] != back[level0]))


@pytest.mark.parametrize("dims", DIMS)
def test_lost_codes_count_the_codes_with_any_plane_lost(dims):
    in_step, lost = planes_of(dims, 0)
    by_words, lost_by_words = planes_of(dims, 1)
    assert np.array_equal(in_step, by_words) == (dims in SAME)
    assert lost == lost_by_words == P.lost_codes(*dims)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("prog", [False, True])
def test_containers_match_the_oracle(dtype, prog):
    import torch
    assert torch.cuda.is_available()
    from prism_b200 import fields
    h = P.Handle()
    for dims in DIMS:
        nx, ny, nz = dims
        for bound in (1e-3, 1e-6):
            data = fields.make("grf", (nz, ny, nx), dtype, nx + ny)
            comp = P.Compressor(P.Context(nx, ny, nz, np.dtype(dtype), P.REL, bound, prog), h)
            got = comp.compress_pipeline(torch.from_numpy(data).cuda()).cpu().numpy().tobytes()
            want, _, _ = O.compress(data, 1, bound, 0 if prog else 1, force=O.intp(*comp.flags))
            assert got == want, (dims, bound)
    h.close()
