"""Matmul on CTA pairs (tiles of 256 x 256): an odd number of 128-row tiles, a ragged last column tile, a depth that is no
multiple of 64, and last rounds that are whole, cut in halves (the most and the fewest items) or too full to be cut."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from oracle import binding as ob  # noqa: E402
from nncv_b200._lib import BF16, F16, F32  # noqa: E402
import gpu_util as G  # noqa: E402


@pytest.mark.parametrize("m,n,k", [(9472, 512, 64), (9600, 512, 72), (2400, 2056, 200), (9300, 768, 136), (4800, 1536, 328)])
@pytest.mark.parametrize("ab", [F16, BF16])
@pytest.mark.parametrize("c_dt", ["same", "f32"])
def test_matmul_on_pairs(m, n, k, ab, c_dt):
    r = np.random.default_rng(m + n + k)
    a = r.uniform(-1, 1, (m, k)).astype(np.float32)
    b = r.uniform(-1, 1, (k, n)).astype(np.float32)
    bias = r.standard_normal(n).astype(np.float32)
    c, ar, br = G.matmul(a, b, ab, ab if c_dt == "same" else F32, bias, True)
    ref = ob.matmul(ar, br, bias, True, acc64=True)
    assert np.isfinite(c).all()
    # fp32 sums of k terms in another order; a 16-bit result is rounded once more, by half a unit in the last place
    bound = 1e-5 + (0 if c_dt == "f32" else 2.0 ** -11 if ab == F16 else 2.0 ** -8)
    assert G.rel_l2(c, ref) <= bound
    assert np.abs(c - ref).max() <= 2 * bound * np.abs(ref).max()
