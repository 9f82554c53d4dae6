"""CPU check of the build's FP32 estimate of a loose box's location (octree_gb300/csrc/otg_build.cu:
box_key_estimate): where it decides, the key must be the reference's. The estimate is restated in numpy
FP32 arithmetic and compared with the oracle's keys for boxes whose centres lie on cell boundaries and
whose sizes lie on powers of two of the cell, a few ulps and fractions of the margin either side."""
import numpy as np
import pytest

from _oracle_lib import KIND_LOOSE_BOXES, oracle
from test_cell_estimate_margin import LOW, SIZE, approx_f

F = np.float32


def part1by2(v):
    v = v.astype(np.uint64)
    for s, m in ((32, 0x1F00000000FFFF), (16, 0x1F0000FF0000FF), (8, 0x100F00F00F00F00F), (4, 0x10C30C30C30C30C3), (2, 0x1249249249249249)):
        v = (v | (v << np.uint64(s))) & np.uint64(m)
    return v


def estimate_keys(boxes, lo, hi, depth, margin_scale=1.0):
    """(decided, key) per box."""
    res, cells = 1 << depth, (1 << depth) + 2
    if boxes.dtype == np.float32:
        size = (hi - lo).astype(F)
        rast = (F(res) / size).astype(F)
        rast_d = rast.astype(np.float64)
        c = boxes
    else:
        size = hi - lo
        rast_d = res / size
        rast = rast_d.astype(F)
        c = approx_f(boxes.reshape(-1)).reshape(boxes.shape)
    M = np.maximum(np.abs(lo.astype(np.float64)), np.abs(hi.astype(np.float64)))
    md = rast_d * M * 2.0**-22 + cells * 2.0**-22 + 2.0**-20
    m32 = md.astype(F)
    m32 = np.where(m32.astype(np.float64) < md, np.nextafter(m32, F(np.inf)), m32)
    m32 = np.where(md < 0.25, m32 * F(margin_scale), F(2)).astype(F)
    a, b = ((c[:, :3] - lo.astype(F)) * rast).astype(F), ((c[:, 3:] - lo.astype(F)) * rast).astype(F)
    top = F(res) - m32
    ok = ((a > m32) & (a < top) & (b > m32) & (b < top)).all(1)
    est = (F(0.5) * (a + b)).astype(F)
    r = np.maximum((b - a).max(1), F(0)).astype(F)
    m = m32.max()
    ok &= m < F(0.25)
    ex = np.where(r > 0, np.frexp(np.where(r > 0, r, F(1)))[1] - 1, -126)
    big = r >= F(0.5)
    p = np.ldexp(F(1), np.where(big, ex, 0)).astype(F)
    ok &= np.where(big, ((r - p) > F(3) * m) & ((F(2) * p - r) > F(3) * m), F(0.5) + F(3) * m < F(1))
    level = np.where(big, ex + 1, 0)
    scale = np.ldexp(F(1), -level).astype(F)[:, None]
    g_f = (est * scale).astype(F)
    ok &= (g_f >= 0).all(1)
    g = np.where(g_f >= 0, np.trunc(g_f), 0)
    f = (g_f - g.astype(F)).astype(F)
    ms = (F(2) * m * scale).astype(F)
    ok &= ((f > ms) & (f < F(1) - ms)).all(1)
    g = g.astype(np.uint64) << np.maximum(level, 0).astype(np.uint64)[:, None]
    loc = part1by2(g[:, 0]) | (part1by2(g[:, 1]) << np.uint64(1)) | (part1by2(g[:, 2]) << np.uint64(2))
    return ok, (loc << np.uint64(5)) | (depth - np.clip(level, 0, depth)).astype(np.uint64)


def make_boxes(rng, depth, offset, dtype, n=30_000):
    lo = offset + LOW
    w = SIZE / (1 << depth)
    level = rng.integers(0, depth, n)[:, None]
    cell = w * 2.0**level
    margin = (SIZE + abs(offset)) * 2.0**-22 + SIZE * 2.0**-22
    near = lambda: rng.choice([0.0, 0.0, 1e-16 * SIZE, -1e-16 * SIZE, 0.5 * margin, -0.5 * margin, 1.5 * margin, -1.5 * margin, 4 * margin], (n, 3))
    size = np.where(rng.random((n, 3)) < 0.5, cell, cell * rng.random((n, 3))) + near()
    centre = lo + np.round(rng.random((n, 3)) * (SIZE / cell)) * cell + near()
    centre = np.where(rng.random((n, 1)) < 0.5, centre, lo + rng.random((n, 3)) * SIZE)
    b = np.concatenate([centre - size / 2, centre + size / 2], 1)
    keep = (b[:, :3] >= lo - SIZE * 1e-9).all(1) & (b[:, 3:] <= lo + SIZE * (1 + 1e-9)).all(1)
    return b[keep].astype(dtype)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("depth", [3, 7, 10, 12])
@pytest.mark.parametrize("offset", [0.0, 819.0, -5000.0, 1e6])
def test_decided_keys_match_the_oracle(dtype, depth, offset):
    rng = np.random.default_rng(depth * 11 + int(abs(offset)) % 1000)
    b = make_boxes(rng, depth, offset, dtype)
    space = np.array([offset + LOW] * 3 + [offset + LOW + SIZE] * 3, dtype)
    for box in (None, space):
        lo = b[:, :3].min(0) if box is None else box[:3]
        hi = b[:, 3:].max(0) if box is None else box[3:]
        ok, key = estimate_keys(b, lo, hi, depth)
        ref = oracle().create(b, KIND_LOOSE_BOXES, depth, box, 16).location_keys()
        bad = ok & (key != ref)
        assert not bad.any(), f"{int(bad.sum())} of {int(ok.sum())} decided keys differ, e.g. {b[np.argmax(bad)]}"
        if offset == 0.0 and depth >= 7:  # (at depth 3 most of these boxes lie on boundaries)
            assert ok.mean() > 0.1
        if offset == 1e6 and dtype == np.float64 and depth >= 12:
            assert not ok.any()


def test_the_inputs_need_the_margin():
    rng = np.random.default_rng(3)
    b = make_boxes(rng, 10, 819.0, np.float64)
    ok, key = estimate_keys(b, b[:, :3].min(0), b[:, 3:].max(0), 10, margin_scale=0.0)
    ref = oracle().create(b, KIND_LOOSE_BOXES, 10, None, 16).location_keys()
    assert (ok & (key != ref)).any()
