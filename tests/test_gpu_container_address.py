"""Containers and streams at addresses that are not multiples of 8: the size
table is then read one entry at a time and the trailer written byte by byte."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(100, 90, 77), (300, 301, 1), (40, 23, 17)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_container_at_an_offset(dims, dtype):
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    from prism_b200 import fields
    nx, ny, nz = dims
    data = torch.from_numpy(fields.make("sinusoid", (nz, ny, nx), dtype, 5)).cuda()
    comp = P.Compressor(P.Context(nx, ny, nz, np.dtype(dtype), P.REL, 1e-4, False))
    cap = comp.max_container_size()
    want = comp.compress_pipeline(data).clone()
    values = comp.decompress_pipeline(want).clone()
    for shift in (2, 4, 6, 8, 12):
        buf = torch.zeros(cap + 64, dtype=torch.uint8, device="cuda")
        assert buf.data_ptr() % 16 == 0
        got = comp.compress_pipeline(data, buf[shift:shift + cap])
        assert torch.equal(got, want), shift
        assert not buf[:shift].any()
        if shift % np.dtype(dtype).itemsize == 0:
            assert torch.equal(comp.decompress_pipeline(got), values), shift
        else:  # the anchors are read in place
            with pytest.raises(P.PrismError):
                comp.decompress_pipeline(got)


@pytest.mark.parametrize("dims", DIMS)
def test_lossless_stream_at_an_offset(dims):
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    l, h = P.lib(), P.Handle()
    n = int(l.prism_plane_buffer_size(*dims))
    rng = np.random.default_rng(2)
    planes = rng.integers(0, 256, n, dtype=np.uint8)
    planes[rng.random(n) < 0.6] = 0
    planes[n // 2:] = 0
    d_planes = torch.from_numpy(planes).cuda()
    cap = n + 2 * (n // 16384 + 256) + 64
    st, size = C.c_void_p(torch.cuda.current_stream().cuda_stream), C.c_uint64()
    streams = []
    for shift in (0, 2, 4, 6):
        buf = torch.zeros(cap + 64, dtype=torch.uint8, device="cuda")
        at = C.c_void_p(buf.data_ptr() + shift)
        assert l.prism_lossless_encode(h.ptr, C.c_void_p(d_planes.data_ptr()), *dims, at, cap, C.byref(size), None,
                                       st) == 0
        streams.append(buf[shift:shift + size.value].cpu().numpy().tobytes())
        out = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
        assert l.prism_lossless_decode(h.ptr, at, *dims, None, None, C.c_void_p(out.data_ptr()), st) == 0
        assert np.array_equal(out.cpu().numpy(), planes), shift
    assert len(set(streams)) == 1
    h.close()
