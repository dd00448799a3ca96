"""Encoding and decoding that skip all-zero (and unselected) chunks.

The encoder does not read chunks whose shuffle items had no nonzero byte.

The decoder leaves such chunks of the plane buffer alone but for their ends,
and the inverse shuffle skips the rows that lie in them.  The host chunk
table and the device plane placement drift apart, so rows straddle chunk
boundaries: the shapes have planes of one chunk, of a few, and last chunks of
a handful of bytes; the bounds leave few or most planes all-zero, and a
handle is reused so that its plane buffer holds other bytes than zeros."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# chunks a level-0 plane (bytes of the last): 17 (13400), 2 (192), 3 (664); 2-D
# 4; 1-D 2; one chunk a plane
SHAPES = [(200, 130, 97), (65, 65, 36), (512, 24, 25), (801, 813, 1), (300007, 1, 1), (40, 23, 17)]


def field(dims, dtype, seed):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    v = np.sin(0.05 * x + 0.03 * y) * np.cos(0.04 * z)
    v[rng.random(v.shape) < 1e-3] += 100.0  # a few large codes: sparse chunks in every plane
    v[:, : ny // 2] = 0.25                  # and runs of zeros
    return v.astype(dtype)


@pytest.fixture(scope="module")
def env():
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    return torch, P, P.Handle()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", SHAPES)
def test_round_trip_matches_oracle(env, dims, dtype):
    torch, P, h = env
    data = field(dims, dtype, sum(dims))
    for bound in (1e-6, 1e-3):  # the tight one first: it fills the plane buffer
        ctx = P.Context(*dims, np.dtype(dtype), P.REL, bound, False)
        comp = P.Compressor(ctx, h)
        cont = comp.compress_pipeline(torch.from_numpy(data).cuda()).clone()
        want, _, _ = O.compress(data, ctx.error_mode, bound, 1, force=O.intp(*comp.flags))
        assert cont.cpu().numpy().tobytes() == want, bound
        got = comp.decompress_pipeline(cont).cpu().numpy()
        want = O.decompress(cont.cpu().numpy().tobytes(), ctx.shape, dtype, ctx.error_mode, bound)
        assert np.array_equal(got.view(np.uint8), want.view(np.uint8)), bound


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("dims", SHAPES)
def test_progressive_matches_oracle(env, dims, exact):
    torch, P, h = env
    data = field(dims, np.float64, 1 + sum(dims))
    ctx = P.Context(*dims, np.dtype(np.float64), P.REL, 1e-6, True)
    comp = P.Compressor(ctx, h)
    cont = comp.compress_pipeline(torch.from_numpy(data).cuda()).clone()
    host = cont.cpu().numpy().tobytes()
    prog, st = comp.progressive(cont), O.ProgressiveState()
    prog.exact(exact)
    for target in (1e-2, 1e-3, 1e-6):
        got = prog.step(target).cpu().numpy()
        want, (b, e, ml) = O.progressive_step(host, ctx.shape, ctx.dtype, ctx.error_mode, ctx.bound, target, st,
                                              exact=exact)
        assert prog.state()[1] == e
        assert np.array_equal(got.view(np.uint8), want.view(np.uint8)), target
    prog.close()
