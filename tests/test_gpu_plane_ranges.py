"""prism_lossless_decode with plane ranges that reach past a level's 32
planes: the chunks of no other level are decoded."""
import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [3, 2, 1, 0])
@pytest.mark.parametrize("lo,hi", [(0, 33), (0, 40), (20, 64), (-3, 32), (32, 40), (40, 50), (-5, -1)])
def test_ranges_past_a_levels_planes(level, lo, hi):
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    l, h = P.lib(), P.Handle()
    dims = (96, 80, 64)
    g = O.geometry(*dims, 4)
    n = int(l.prism_plane_buffer_size(*dims))
    planes = np.random.default_rng(7).integers(1, 256, n, dtype=np.uint8)  # no byte zero: every chunk coded
    d_planes = torch.from_numpy(planes).cuda()
    cap = n + 2 * (n // 16384 + 256) + 64
    d_stream = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    st, size = C.c_void_p(torch.cuda.current_stream().cuda_stream), C.c_uint64()
    assert l.prism_lossless_encode(h.ptr, C.c_void_p(d_planes.data_ptr()), *dims, C.c_void_p(d_stream.data_ptr()), cap,
                                   C.byref(size), None, st) == 0
    begin, end = (C.c_int * 4)(), (C.c_int * 4)()
    begin[3 - level], end[3 - level] = lo, hi
    out = torch.zeros(n, dtype=torch.uint8, device="cuda")
    assert l.prism_lossless_decode(h.ptr, C.c_void_p(d_stream.data_ptr()), *dims, begin, end,
                                   C.c_void_p(out.data_ptr()), st) == 0
    stride = [int(v) for v in g.hastride]
    at = sum(32 * stride[i] for i in range(level + 1, 4))
    want = np.zeros(n, dtype=np.uint8)
    s, e = at + min(max(lo, 0), 32) * stride[level], at + min(max(hi, 0), 32) * stride[level]
    want[s:e] = planes[s:e]
    assert np.array_equal(out.cpu().numpy(), want)
    h.close()
