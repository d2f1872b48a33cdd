"""fp32 convolutions of stride 1 on 128 x 64 tiles: one box of pixels for a whole column of the filter, against a copy for every tap and
against 64 bits, at the edges of tiles, images and split reductions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200 import runtime as rt  # noqa: E402
from nncv_b200._lib import F32, check, lib  # noqa: E402
import gpu_util as G  # noqa: E402


@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("case", [
    # n, c, h, w, k, r, pad: columns of 8, 16 and 56 pixels; images one below the other (7 x 7, 5 x 5, 3 x 3); a single row or column
    (2, 64, 16, 8, 64, 3, 1), (1, 64, 17, 9, 64, 3, 1), (3, 72, 14, 14, 68, 3, 1), (1, 64, 56, 56, 64, 3, 1), (5, 64, 7, 7, 128, 3, 1),
    (9, 8, 5, 5, 12, 3, 1), (7, 136, 3, 3, 64, 3, 1), (1, 64, 1, 200, 8, 3, 1), (1, 40, 131, 3, 100, 3, 1), (1, 8, 1, 1, 4, 3, 1),
    # other filters and pads; more tiles than SMs
    (2, 64, 20, 21, 64, 5, 2), (2, 64, 12, 19, 64, 3, 0), (2, 64, 7, 7, 64, 3, 2), (3, 128, 9, 11, 64, 7, 3), (40, 16, 28, 28, 64, 3, 1),
])
def test_one_box_for_a_column_of_the_filter(case, splits):
    n, c, h, w, k, r, pad = case
    if splits > r * r * -(-c // 64):
        pytest.skip("more CTAs than blocks of 64 channels")
    g = np.random.default_rng(sum(case))
    x = g.standard_normal((n, c, h, w)).astype(np.float32)
    wt = (g.standard_normal((k, c, r, r)) * np.sqrt(2.0 / (c * r * r))).astype(np.float32)
    conv = G.Conv(wt, 1, pad, F32)
    got = []
    try:
        for way in (2, 1):
            check(lib().nncv_b200_conv_set_tile(conv.h, 64, splits, way))
            check(lib().nncv_b200_profile(1))
            y, _ = conv.run(x)
            made = [q["bn"] for q in rt.profile_records() if q["kind"] == 1]
            check(lib().nncv_b200_profile(0))
            assert made == [640 + splits + (1000 if way == 2 else 0)]   # what ran: boxes for columns, copies for taps
            got.append(y)
    finally:
        conv.close()
    ref = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(wt).double(), padding=pad).numpy()
    # the steps of the large products are cut to 24 bits (2^-23 of a step), their running sum rounded (2^-24 each, like a random walk)
    bound = 4 * 2.0 ** -23 + 2.0 ** -24 * np.sqrt(r * r * np.ceil(c / 64))
    for y in got:
        assert np.isfinite(y).all() and G.rel_l2(y, ref) <= bound
    assert G.rel_l2(got[0], got[1]) <= bound
    assert lib().nncv_b200_device_status() == 0


def test_a_box_keeps_infinities_where_they_belong():
    """An infinite pixel reaches the outputs under its window and no others: images lie one below the other in a tile."""
    x = np.ones((4, 64, 7, 7), np.float32)
    x[1, 5, 6, 3] = np.inf
    conv = G.Conv(np.full((64, 64, 3, 3), 0.125, np.float32), 1, 1, F32)
    try:
        check(lib().nncv_b200_conv_set_tile(conv.h, 64, 1, 2))
        check(lib().nncv_b200_profile(1))
        y, _ = conv.run(x)
        made = [q["bn"] for q in rt.profile_records() if q["kind"] == 1]
        check(lib().nncv_b200_profile(0))
    finally:
        conv.close()
    assert made == [1641]
    want = np.zeros((4, 64, 7, 7), bool)
    want[1, :, 5:7, 2:5] = True
    assert np.array_equal(np.isinf(y), want) and not np.isnan(y).any()


@pytest.mark.parametrize("case", [(2, 128, 9, 9, 64, 1, 1), (2, 64, 9, 9, 64, 3, 2), (1, 64, 40, 24, 64, 19, 1)])
def test_what_boxes_do_not_fit_is_copied_by_taps(case):
    """1x1 filters, strides, and columns too long for two boxes in shared memory."""
    n, c, h, w, k, r, stride = case
    g = np.random.default_rng(sum(case))
    x, wt = g.standard_normal((n, c, h, w)).astype(np.float32), (g.standard_normal((k, c, r, r)) / r).astype(np.float32)
    conv = G.Conv(wt, stride, r // 2, F32)
    try:
        check(lib().nncv_b200_conv_set_tile(conv.h, 64, 1, 2))
        check(lib().nncv_b200_profile(1))
        y, _ = conv.run(x)
        made = [q["bn"] for q in rt.profile_records() if q["kind"] == 1]
        check(lib().nncv_b200_profile(0))
    finally:
        conv.close()
    assert made == [641]
    ref = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(wt).double(), stride=stride, padding=r // 2).numpy()
    assert G.rel_l2(y, ref) <= 4 * 2.0 ** -23 + 2.0 ** -24 * np.sqrt(4 * r * r)


@pytest.mark.parametrize("bn,splits", [(64, 1), (64, 4), (128, 1), (128, 2), (128, 8)])
@pytest.mark.parametrize("case", [
    # n, c, h, w, k, r, stride: one block of 64 channels, two, four, as many as the rings hold and more, a multiple of neither ring
    (2, 64, 9, 9, 128, 1, 1), (2, 128, 9, 9, 132, 1, 1), (1, 232, 5, 7, 260, 1, 1), (2, 64, 20, 21, 128, 3, 2), (3, 136, 13, 11, 192, 3, 2), (2, 512, 7, 7, 256, 3, 1),
    # more tiles than SMs: the rings go on from tile to tile
    (40, 72, 28, 28, 256, 1, 1), (24, 64, 57, 55, 128, 3, 2), (70, 48, 15, 15, 320, 1, 2),
])
def test_a_copy_for_every_tap(case, bn, splits):
    n, c, h, w, k, r, stride = case
    if splits > r * r * -(-c // 64):
        pytest.skip("more CTAs than blocks of 64 channels")
    g = np.random.default_rng(sum(case))
    x = g.standard_normal((n, c, h, w)).astype(np.float32)
    wt = (g.standard_normal((k, c, r, r)) * np.sqrt(2.0 / (c * r * r))).astype(np.float32)
    conv = G.Conv(wt, stride, r // 2, F32)
    try:
        check(lib().nncv_b200_conv_set_tile(conv.h, bn, splits, 1))
        check(lib().nncv_b200_profile(1))
        y, _ = conv.run(x)
        made = [q["bn"] for q in rt.profile_records() if q["kind"] == 1]
        check(lib().nncv_b200_profile(0))
        again, _ = conv.run(x)
    finally:
        conv.close()
    assert made == [10 * bn + splits] and np.array_equal(y, again)
    ref = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(wt).double(), stride=stride, padding=r // 2).numpy()
    assert np.isfinite(y).all() and G.rel_l2(y, ref) <= 4 * 2.0 ** -23 + 2.0 ** -24 * np.sqrt(4 * r * r * np.ceil(c / 64))
    assert lib().nncv_b200_device_status() == 0
