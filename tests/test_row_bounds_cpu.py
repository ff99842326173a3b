"""The geometry passes' one-row test (row_empty in swegl_gb300/csrc/raster.cu)
is safe: a float32 emulation of fill_triangle_2's edge set-up finds no pixel in
the row of any triangle the test removes.  Triangles of one row are built with
a crossing of the row within 1e-10 .. 1e-4 (relative) of a pixel column, widths
from 1e-3 to 3e4 and |x| up to 3e4, edges as flat as the row allows, vertices
on the row; the reciprocal is off by up to one unit in the last place either
way, as the hardware's.  With eps = 0 the same emulation does find pixels, so
the margin is what makes it safe."""
import math

import numpy as np

from test_walk_bounds_cpu import _ceil, f, walk_spans


def row_empty(xs, ys, rng, margin=True):
    lo_y, hi_y = min(ys), max(ys)
    y = f(_ceil(lo_y))
    mx = f(max(abs(x) for x in xs))
    if not (f(y + f(1.0)) >= hi_y and mx < f(2.0 ** 20) and abs(y) < f(2.0 ** 20)):
        return False
    rows = f(_ceil(hi_y) - _ceil(lo_y))
    eps = f(f(f(rows + f(32.0)) * f(2.0 ** -23)) * f(mx + f(1.0))) if margin else f(0.0)
    lo, hi, total = f(np.inf), f(-np.inf), f(0.0)
    for a, b in ((0, 1), (1, 2), (2, 0)):
        d = f(ys[b] - ys[a])
        if (ys[a] <= y) != (ys[b] <= y):
            r = f(f(1.0) / d)
            r = np.nextafter(r, f(rng.choice([-np.inf, np.inf]))) if rng.uniform() < 0.5 else r
            x = f(xs[a] + f(f(f(y - ys[a]) * f(xs[b] - xs[a])) * r))
            lo, hi, total = min(lo, x), max(hi, x), f(total + x)
    return abs(total) < f(2.0 ** 22) and _ceil(f(lo - eps)) >= f(hi + eps)


def triangles(n, rng):
    for _ in range(n):
        row = int(rng.integers(-50, 2000))
        up, down = 10.0 ** rng.uniform(-6, 0), 10.0 ** rng.uniform(-6, 0)
        ys = [f(row - up * rng.uniform(0, 0.99)), f(row + down * rng.uniform(0.001, 0.99)),
              f(rng.uniform(row - 0.99 * up, row + 0.99 * down))]
        if rng.uniform() < 0.2:
            ys[int(rng.integers(0, 3))] = f(row)
        col = math.floor(10.0 ** rng.uniform(0, 4.5)) * rng.choice([-1, 1])
        width = 10.0 ** rng.uniform(-3, 4.5)
        xs = [rng.uniform(-width, width) for _ in range(3)]
        # shifted so that one crossing of the row lies near the column
        edges = [(a, b) for a, b in ((0, 1), (1, 2), (2, 0)) if (ys[a] <= row) != (ys[b] <= row)]
        if len(edges) != 2 or not min(ys) <= row < max(ys) or math.ceil(max(ys)) != row + 1 or math.ceil(min(ys)) != row:
            continue
        a, b = edges[int(rng.integers(0, 2))]
        at = xs[a] + (row - float(ys[a])) * (xs[b] - xs[a]) / (float(ys[b]) - float(ys[a]))
        gap = 10.0 ** rng.uniform(-10, -4) * max(1.0, abs(col)) * rng.choice([-1, 1])
        yield [f(x - at + col + gap) for x in xs], ys


def test_removed_triangles_have_no_pixel():
    rng = np.random.default_rng(3)
    removed = 0
    for xs, ys in triangles(60000, rng):
        if row_empty(xs, ys, rng):
            removed += 1
            assert all(a >= b for (a, b) in walk_spans(list(zip(xs, ys)))), (xs, ys)
    assert removed > 3000


def test_without_the_margin_rows_get_pixels():
    rng = np.random.default_rng(4)
    hits = sum(any(a < b for (a, b) in walk_spans(list(zip(xs, ys)))) for xs, ys in triangles(60000, rng)
               if row_empty(xs, ys, rng, margin=False))
    assert hits > 0
