"""Error statistics over one CTA, fewer than a fold's 256 partials, more, and
remainders of the four-value loop: exact extremes and first index, and the
squared-error sum against numpy's in long double.  The kernel adds n terms in
a tree of depth at most n / 2^18 + 32 per path, each rounding within
2^-53 of a partial sum below the total."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 2, 255, 257, 40_001, 256 * 256, 256 * 300 + 1, 256 * 1184 * 4 + 3, 3_000_017])
def test_statistics(n, dt):
    import torch
    import prism_b200 as P
    assert torch.cuda.is_available()
    rng = np.random.default_rng(n)
    ori = rng.normal(0, 1, n).astype(dt)
    dat = (ori + rng.normal(0, 1e-3, n)).astype(dt)
    s = P.Handle().statistics(torch.from_numpy(ori).cuda(), torch.from_numpy(dat).cuda())
    err = np.abs((dat - ori).astype(np.float64))
    assert s["max_err"] == err.max() and s["max_err_index"] == int(np.argmax(err))
    assert s["min"] == float(ori.min()) and s["max"] == float(ori.max())
    l2 = float(np.sum(err.astype(np.longdouble) ** 2))
    assert abs(s["l2"] - l2) <= (n / 2 ** 18 + 32) * 2.0 ** -53 * l2
