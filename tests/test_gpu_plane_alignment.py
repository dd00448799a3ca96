"""prism_bitshuffle of fields within one shuffle block (no 4-byte plane
stores) into a plane buffer at any byte address."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(5, 3, 2), (17, 9, 5), (16, 16, 16), (33, 20, 21), (100, 37, 1), (1023, 1, 1)])
def test_planes_at_any_address(dims):
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    l, h = P.lib(), P.Handle()
    ncodes, n = int(l.prism_code_buffer_len(*dims)), int(l.prism_plane_buffer_size(*dims))
    rng = np.random.default_rng(sum(dims))
    codes = torch.from_numpy(rng.integers(-2 ** 31, 2 ** 31, ncodes, dtype=np.int64).astype(np.int32)).cuda()
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    got = []
    for shift in range(4):
        buf = torch.zeros(n + 64, dtype=torch.uint8, device="cuda")
        assert l.prism_bitshuffle(h.ptr, C.c_void_p(codes.data_ptr()), *dims, 1,
                                  C.c_void_p(buf.data_ptr() + shift), st) == 0
        got.append(buf[shift:shift + n].cpu().numpy())
        assert not buf[:shift].any() and not buf[shift + n:].any()
    for g in got[1:]:
        assert np.array_equal(g, got[0])
    h.close()
