"""The beam grid's candidates pair for pair: the reference's walk (Grid.hxx:322-398) and the whole predicate
(PhotonBeam.hxx:238-296) for every entry of every visited cell, in the reference's FP32 operations, here in
numpy on the cell lists that the build made.  The gather's first checks (on 16-byte lines) may drop no pair of
these, so counts and hashes are equal."""
import numpy as np
import pytest

from smallupbp_b200 import engine
from smallupbp_b200 import workload as W

F = np.float32


def header(w, res):
    """The grid's box, resolution, cell size and its inverse (Grid.hxx:222-241)."""
    o, d, n = w["beam_origin"], w["beam_direction"], w["beam_length"][:, None]
    r = F(w["params"]["radius_bb1d"][0])
    sq = d * d
    m = np.sqrt(np.stack([sq[:, 1] + sq[:, 2], sq[:, 0] + sq[:, 2], sq[:, 0] + sq[:, 1]], 1))
    e, rm = o + d * n, r * m
    lo = np.minimum(o - rm, e - rm).min(axis=0)
    hi = np.maximum(o + rm, e + rm).max(axis=0)
    ext = hi - lo
    size = ext.max() / F(res)
    cells = (ext / size).astype(np.uint32).astype(np.int64) + 1
    cell = ext / cells.astype(F)
    return lo, hi, cells, cell, F(1) / cell


def dot(a, b):
    return (a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1]) + a[:, 2] * b[:, 2]


def accepted(o1, d1, tmin, tmax, o2, d2, length, r):
    """testIntersectionBeamBeam and the radius test, one pair per row."""
    c = np.stack([d1[:, 1] * d2[:, 2] - d1[:, 2] * d2[:, 1], d1[:, 2] * d2[:, 0] - d1[:, 0] * d2[:, 2],
                  d1[:, 0] * d2[:, 1] - d1[:, 1] * d2[:, 0]], 1)
    s2 = dot(c, c)
    ad = dot(o2 - o1, c)
    b = dot(d1, d2)
    m1 = b * b - F(1)
    e = dot(d2, o1) - dot(d2, o2)
    d1o1, d1o2 = dot(d1, o1), dot(d1, o2)
    with np.errstate(all="ignore"):
        t1 = ((d1o1 - d1o2) - b * e) / m1
        t2 = ((t1 + d1o1) - d1o2) / b
        dist = np.abs(ad) / np.sqrt(s2)
        return (~(ad * ad >= r * r * s2) & ~((m1 < F(1e-5)) & (m1 > F(-1e-5))) & ~((t1 <= tmin) | (t1 >= tmax)) &
                ~((t2 <= 0) | (t2 >= length) | np.isnan(t2)) & ~(r < dist))


def mix64(i):
    z = i.astype(np.uint64) + np.uint64(1) + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def candidates(w, res, grid):
    lo, hi, cells, cell, inv = header(w, res)
    assert len(grid["cells"]) == (cells + 1).prod() + 1
    r = F(w["params"]["radius_bb1d"][0])
    count = np.zeros(len(w["sq_flags"]), np.int64)
    hashes = np.zeros(len(w["sq_flags"]), np.uint64)
    # one row per scattering segment of a query
    q = np.repeat(np.arange(len(count)), w["sq_seg_count"])
    s = np.concatenate([np.arange(b, b + n) for b, n in zip(w["sq_seg_begin"], w["sq_seg_count"])])
    use = (w["seg_medium"][s] == 1) & ((w["sq_flags"][q] & W.Q_BB1D) != 0)
    q, s = q[use], s[use]
    o, d = w["sq_origin"][q], w["sq_direction"][q]
    with np.errstate(all="ignore"):
        i = F(1) / d
        l1, l2 = (lo - o) * i, (hi - o) * i
        l1, l2 = np.where(np.isnan(l1), F(np.inf), l1), np.where(np.isnan(l2), F(np.inf), l2)
        lmax, lmin = np.maximum(l1, l2).min(axis=1), np.minimum(l1, l2).max(axis=1)
    mint, maxt = w["seg_dist_min"][s], w["seg_dist_max"][s]
    tmn, tmx = np.where(lmin < mint, mint, lmin), np.where(lmax > maxt, maxt, lmax)
    go = (lmax >= lmin) & (tmx > tmn)
    q, o, d, i, tmx, t = q[go], o[go], d[go], i[go], tmx[go], tmn[go]
    e = ((o + d * t[:, None]) - lo) * inv
    p = np.clip(np.trunc(e).astype(np.int64), 0, cells - 1)
    up = d >= 0
    step = np.where(up, 1, -1)
    end = np.where(up, cells, -1)
    delta = np.abs(cell * i)
    left = ((p + up).astype(F) - e) * i * cell
    shift = np.array([1, cells[0], cells[0] * cells[1]])
    at = (p * shift).sum(axis=1)
    rows = np.arange(len(q))
    for _ in range(int(cells.sum()) + 3):
        x, y, z = left.T
        ax = np.where(x < y, np.where(x < z, 0, 2), np.where(y < z, 1, 2))
        la = left[np.arange(len(ax)), ax]
        tn = t + la
        hi_t = np.where(tmx < tn, tmx, tn)
        begin, n = grid["cells"][at].astype(np.int64), grid["cells"][at + 1].astype(np.int64)
        n = n - begin
        k = np.repeat(np.arange(len(at)), n)
        beam = grid["beams"][np.arange(n.sum()) - np.repeat(n.cumsum() - n, n) + np.repeat(begin, n)]
        row = rows[k]
        ok = accepted(o[row], d[row], t[k], hi_t[k], w["beam_origin"][beam], w["beam_direction"][beam],
                      w["beam_length"][beam], r) & (w["beam_medium_id"][beam] == 1)
        np.add.at(count, q[row[ok]], 1)
        np.add.at(hashes, q[row[ok]], mix64(beam[ok]))
        # the next cell
        t = tn
        left = left - la[:, None]
        left[np.arange(len(ax)), ax] = delta[rows, ax]
        p[np.arange(len(ax)), ax] += step[rows, ax]
        at = at + shift[ax] * step[rows, ax]
        on = (p[np.arange(len(ax)), ax] != end[rows, ax]) & (t < tmx)
        t, tmx, left, p, at, rows = t[on], tmx[on], left[on], p[on], at[on], rows[on]
        if not len(rows):
            break
    assert not len(rows)
    return count, hashes


@pytest.mark.gpu
@pytest.mark.parametrize("res,shift", [(1, 0.0), (7, 0.0), (64, 0.0), (7, 32.0)])
def test_the_gather_takes_every_pair_of_the_predicate(res, shift):
    w = W.generate(W.cube_scene("lines", 40, 30, 400, 6, 0.04, techniques=W.BPT | W.BB1D), 0)
    for k in ("lv_position", "beam_origin", "sq_origin"):
        w[k] = (w[k] + F(shift)).astype(F)
    for mode in (engine.MODE_PLAIN, engine.MODE_MIXED):
        with engine.EstimatorStage(0, mode) as st:
            st.set_bb1d_grid(res)
            st.run(w)
            got, grid = st.query_stats(), st.grid_structure()
        if mode == engine.MODE_PLAIN:
            count, hashes = candidates(w, res, grid)
            assert count.sum() > 10000
        np.testing.assert_array_equal(got["count_bb1d"], count)
        np.testing.assert_array_equal(got["hash_bb1d"], hashes)
