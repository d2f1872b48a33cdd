"""Matmul on CTA pairs (tiles of 256 x 256): an odd number of 128-row tiles, a ragged last column tile, a depth that is no
multiple of 64, and last rounds that are whole, cut in halves (the most and the fewest items) or too full to be cut."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200._lib import BF16, F16, F32  # noqa: E402
import gpu_util as G  # noqa: E402


@pytest.mark.parametrize("m,n,k", [(9472, 512, 1024), (9600, 512, 1032), (2400, 2056, 1096), (9300, 768, 1160), (4800, 1536, 1288)])
@pytest.mark.parametrize("ab", [F16, BF16])
@pytest.mark.parametrize("c_dt", ["same", "f32"])
def test_matmul_on_pairs(m, n, k, ab, c_dt):
    r = np.random.default_rng(m + n + k)
    a = r.uniform(-1, 1, (m, k)).astype(np.float32)
    b = r.uniform(-1, 1, (k, n)).astype(np.float32)
    bias = r.standard_normal(n).astype(np.float32)
    c, ar, br = G.matmul(a, b, ab, ab if c_dt == "same" else F32, bias, True)
    ref = np.maximum((torch.from_numpy(ar).cuda().double() @ torch.from_numpy(br).cuda().double()).cpu().numpy() + bias, 0)
    assert np.isfinite(c).all()
    # fp32 sums of k terms in another order; a 16-bit result is rounded once more, by half a unit in the last place
    bound = 1e-5 + (0 if c_dt == "f32" else 2.0 ** -11 if ab == F16 else 2.0 ** -8)
    assert G.rel_l2(c, ref) <= bound
    assert np.abs(c - ref).max() <= 2 * bound * np.abs(ref).max()


@pytest.mark.parametrize("m,n,k", [(16, 64, 512), (1, 72, 520), (50, 200, 1000), (128, 1000, 2048), (300, 104, 4000), (1024, 512, 1096),
                                   (4736, 128, 512), (4737, 128, 512), (2900, 360, 448)])
@pytest.mark.parametrize("ab", [F16, BF16])
@pytest.mark.parametrize("c_dt", ["same", "f32"])
def test_matmul_shared_depth(m, n, k, ab, c_dt):
    """Clusters of two, four or eight CTAs a tile: ragged rows, columns and depth, unequal shares, the most tiles and one
    more; and a matrix whose last tile of 128 rows is mostly empty."""
    r = np.random.default_rng(m + n + k)
    a = r.uniform(-1, 1, (m, k)).astype(np.float32)
    b = r.uniform(-1, 1, (k, n)).astype(np.float32)
    bias = r.standard_normal(n).astype(np.float32)
    for bi, relu in ((None, False), (bias, True)):
        c, ar, br = G.matmul(a, b, ab, ab if c_dt == "same" else F32, bi, relu)
        ref = ar.astype(np.float64) @ br.astype(np.float64)
        if relu:
            ref = np.maximum(ref + bias, 0)
        assert np.isfinite(c).all()
        bound = 1e-5 + (0 if c_dt == "f32" else 2.0 ** -11 if ab == F16 else 2.0 ** -8)
        assert G.rel_l2(c, ref) <= bound
        assert np.abs(c - ref).max() <= 2 * bound * np.abs(ref).max()
