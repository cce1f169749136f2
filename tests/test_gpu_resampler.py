"""The resampler's adjoint against the FP32 oracle: the same products and sums in
the same (target) order, so equal to the bit."""
import numpy as np
import pytest

from gpu_helpers import cu
from oracle import rf_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["ascending", "descending", "random"])
@pytest.mark.parametrize("A,R,S,T", [(1, 9, 2, 1), (2, 17, 31, 33), (3, 8, 64, 512), (1, 5, 33, 513), (2, 3, 100, 1100)])
def test_adjoint_matches_oracle(cuda, A, R, S, T, order):
    from geraf_b200.ops.RFSignalTracer import _C

    rng = np.random.default_rng(T)
    z = np.sort(rng.uniform(0.2, 0.6, (R, S)), axis=1).astype(np.float32)
    tz = rng.uniform(0.15, 0.65, (R, T)).astype(np.float32)
    tz[:, T // 2] = z[:, S // 2]  # on a coarse depth
    if order != "random":
        tz = np.sort(tz, axis=1)[:, ::1 if order == "ascending" else -1]
    tz = tz.copy()
    gon = rng.standard_normal((R, T, 3)).astype(np.float32)
    gos = rng.standard_normal((A, R, T)).astype(np.float32)
    start_n = rng.standard_normal((R, S, 3)).astype(np.float32)
    start_s = rng.standard_normal((A, R, S)).astype(np.float32)
    gn, gs = cu(start_n), cu(start_s)
    _C.BilinearRaysample_backward(cu(gon), cu(gos), cu(z), cu(tz), gn, gs, A, R, S, T)
    rn, rs = orc.bilinear_backward(gon, gos, z, tz, start_n, start_s)
    np.testing.assert_array_equal(gn.cpu().numpy(), rn)
    np.testing.assert_array_equal(gs.cpu().numpy(), rs)
