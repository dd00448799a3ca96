"""Fields with one plane (2-D and 1-D) take the warp-per-tile kernels: codes
and anchors of the predictor, and the reconstruction of the same codes (full
and progressive with the leading levels skipped), against the oracle bit for
bit under forced per-level flags.  Extents at the edges of the 16-point
tiles: 1, 2, one below, at and above a multiple, many tiles, one row."""
import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(2, 1), (1, 2), (16, 16), (17, 17), (15, 33), (3, 100), (129, 70), (257, 18), (1000, 1), (1, 513)]
FLAGS = {
    "md": ([1, 1, 1, 1], [0, 0, 0, 0]),
    "axis": ([0, 0, 0, 0], [0, 0, 0, 0]),
    "axis_rev": ([0, 0, 0, 0], [1, 1, 1, 1]),
    "mixed": ([1, 0, 1, 0], [0, 1, 1, 0]),
}


@pytest.fixture(scope="module")
def env():
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    return torch, P, P.Handle()


@pytest.mark.parametrize("flag_name", list(FLAGS))
@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_flat_predict_and_reconstruct(env, dims, dtype, flag_name):
    torch, P, h = env
    md, rv = FLAGS[flag_name]
    nx, ny = dims
    rng = np.random.default_rng(nx + 7 * ny)
    y, x = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    data = (np.sin(0.11 * x + 0.05 * y) + 0.02 * rng.standard_normal((ny, nx))).astype(dtype)[None]
    eb, l = 1e-3, P.lib()
    flags8 = (C.c_uint8 * 8)(*md, *rv)
    n = int(l.prism_code_buffer_len(nx, ny, 1))
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    codes = torch.zeros(n + 64, dtype=torch.int32, device="cuda")
    anchors = torch.zeros(n, dtype=tdt, device="cuda")
    d_in = torch.from_numpy(data).cuda()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    h.check(l.prism_predict(h.ptr, ptr(d_in), data.itemsize, nx, ny, 1, C.c_double(eb), C.c_double(0.0), flags8,
                            ptr(codes), ptr(anchors), st), "prism_predict")
    o_anchors, o_qc, _ = O.predict(data, eb, md, rv, 0.0)
    na = int(O.geometry(nx, ny, 1, data.itemsize).anchors)
    assert np.array_equal(anchors[:na].cpu().numpy().view(np.uint8), o_anchors.view(np.uint8))
    assert np.array_equal(codes[:nx * ny].cpu().numpy(), o_qc[:nx * ny])
    for maxlevel, prog in [(4, False), (4, True), (1, True)]:
        old = torch.from_numpy(rng.standard_normal(data.shape).astype(dtype)).cuda() if prog else None
        out = old.clone() if prog else torch.empty_like(d_in)  # in place, as a refinement step
        anc = torch.zeros_like(anchors) if prog else anchors
        h.check(l.prism_reconstruct(h.ptr, ptr(codes), ptr(anc), data.itemsize, nx, ny, 1, C.c_double(eb),
                                    C.c_double(0.0), flags8, maxlevel, ptr(out) if prog else None, ptr(out), st),
                "prism_reconstruct")
        want = O.reconstruct(o_qc, anc[:na].cpu().numpy(), data.shape, dtype, eb, md, rv, 0.0, maxlevel,
                             old.cpu().numpy() if prog else None)
        assert np.array_equal(out.cpu().numpy().view(np.uint8), want.view(np.uint8)), (maxlevel, prog)
