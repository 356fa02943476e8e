"""CPU restatement of the layouts the register-held and tensor-core kernels compute
their indices by, for the template instances the sources build (read from them):

* the regions of the multigrid levels (fs_mgreg.cuh) and of the flat solvers
  (fs_flat.cuh): a region is filled with wrapped cells, swept with NaN beyond its
  edge, and what it stores has to cover the level once and equal the sweeps of the
  whole level;
* the operands of the weight gradients (fs_wgrad.cuh), read back through their
  descriptors: the nine taps of the direct correlation;
* the ring of rows of the convolutions (fs_conv.cu): a row is not overwritten before
  the tiles that read it are done.
"""
import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "fluid-sim_gb300" / "csrc"


def _read(name):
    return (CSRC / name).read_text()


# ------------------------------------------------------------------ regions
def sum4(l, r, b, t):
    return ((l + r) + b) + t


def update(c, l, r, b, t, d):
    return c + 1.2 * (0.25 * (sum4(l, r, b, t) - 0.3 * d) - c)


def neighbours(p, edge):
    """(l, r, b, t) of every cell; edge: np.nan, or None for a periodic level"""
    if edge is None:
        return np.roll(p, 1, 1), np.roll(p, -1, 1), np.roll(p, 1, 0), np.roll(p, -1, 0)
    q = np.full((p.shape[0] + 2, p.shape[1] + 2), edge)
    q[1:-1, 1:-1] = p
    return q[1:-1, :-2], q[1:-1, 2:], q[:-2, 1:-1], q[2:, 1:-1]


def half_sweep(p, d, mask, edge):
    return np.where(mask, update(p, *neighbours(p, edge), d), p)


def residual(p, d, edge):
    return d - (sum4(*neighbours(p, edge)) - 4.0 * p) * 3.0


def restrict(r):
    return ((r[0::2, 0::2] + r[0::2, 1::2]) + r[1::2, 0::2] + r[1::2, 1::2]) * 0.25


def prolong(c, ii, jj):
    """the correction at fine cells (jj, ii), coarse indices wrapped"""
    n = c.shape[0]

    def ends(i):
        lo = np.where(i % 2 == 1, i // 2, i // 2 - 1)
        return lo % n, (lo + 1) % n, np.where(i % 2 == 1, 0.25, 0.75)

    x0, x1, fx = ends(ii[None, :])
    y0, y1, fy = ends(jj[:, None])
    top = c[y0, x0] + (c[y0, x1] - c[y0, x0]) * fx
    bot = c[y1, x0] + (c[y1, x1] - c[y1, x0]) * fx
    return top + (bot - top) * fy


def parity(ii, jj):
    return (ii[None, :] + jj[:, None]) & 1


def mg_regions():
    """(side, acc) -> (columns a lane, rows a warp, warps)"""
    src, out = _read("fs_multigrid.cu"), {}
    for args, lane, rows, warps in re.findall(
            r"struct RegionOf(<[^>]*>)? \{\s*typedef MgRegion<(\d+), ([^,]+), (\d+), H> R;", src):
        side = int(re.match(r"<(\d+)", args).group(1)) if args else 64
        for acc in (False, True):
            r = re.match(r"ACC \? (\d+) : (\d+)", rows)
            out[side, acc] = (int(lane), int(r.group(1 if acc else 2)) if r else int(rows), int(warps))
    assert set(out) == {(t, a) for t in (16, 32, 64) for a in (False, True)}
    return out


def mg_shape(region, H):
    cpl, rpw, warps = region
    HX, HY = (H + cpl - 1) // cpl * cpl, (H + 1) & ~1
    return cpl, HX, HY, 32 * cpl, rpw * warps


@pytest.mark.parametrize("n", [66, 72, 100, 126, 132, 264])
@pytest.mark.parametrize("side", [16, 32, 64])
@pytest.mark.parametrize("sweeps", [1, 2, 3])
def test_multigrid_regions(n, side, sweeps):
    if side != 16 and (n % 4 or 2 * side > n):  # not used on this level
        return
    rng = np.random.default_rng(n + side + sweeps)
    x, d = rng.standard_normal((2, n, n))
    coarse = rng.standard_normal((n // 2, n // 2))
    every = np.arange(n)
    # the whole level: down, and up
    down = x
    for s in range(2 * sweeps):
        down = half_sweep(down, d, parity(every, every) == s % 2, None)
    rhs = restrict(residual(down, d, None))
    up = x + prolong(coarse, every, every)
    for s in range(2 * sweeps):
        up = half_sweep(up, d, parity(every, every) == s % 2, None)
    for acc in (False, True):
        for H, is_down in ((2 * sweeps + 1, True), (2 * sweeps, False)):
            if acc and is_down:
                continue
            cpl, HX, HY, RW, RH = mg_shape(mg_regions()[side, acc], H)
            TW, TH = RW - 2 * HX, RH - 2 * HY
            assert n % cpl == 0 and HX % cpl == 0 and HX % 2 == 0 and TW % cpl == 0 and TH % 2 == 0
            stored, out, cr = np.zeros((n, n), int), np.full((n, n), np.nan), np.full((n // 2, n // 2), np.nan)
            for by in range(-(-n // TH)):
                for bx in range(-(-n // TW)):
                    xl, yl = bx * TW - HX + np.arange(RW), by * TH - HY + np.arange(RH)
                    assert (xl[::cpl] % n + cpl <= n).all()  # a lane's columns do not straddle the wrap
                    p, dd = x[np.ix_(yl % n, xl % n)], d[np.ix_(yl % n, xl % n)]
                    if not is_down:
                        p = p + prolong(coarse, xl, yl)
                    for s in range(2 * sweeps):  # the region's first column and row are even
                        p = half_sweep(p, dd, parity(np.arange(RW), np.arange(RH)) == s % 2, np.nan)
                    cols = slice(HX, min(RW - HX, HX + n - bx * TW))
                    rows = slice(HY, min(RH - HY, HY + n - by * TH))
                    at = np.ix_(yl[rows], xl[cols])
                    stored[at] += 1
                    out[at] = p[rows, cols]
                    if is_down:
                        r = restrict(residual(p, dd, np.nan)[rows, cols])
                        cr[np.ix_(yl[rows][::2] // 2, xl[cols][::2] // 2)] = r
            assert (stored == 1).all()
            np.testing.assert_array_equal(out, down if is_down else up)
            if is_down:
                np.testing.assert_array_equal(cr, rhs)


FLAT = sorted({tuple(map(int, t)) for t in re.findall(r"flat_t<(\d+), (\d+), (\d+), (\d+), MODE>", _read("fs_flat.cu"))})


@pytest.mark.parametrize("tile", FLAT)
@pytest.mark.parametrize("ny, nx", [(16, 16), (17, 20), (40, 130), (133, 65)])
def test_flat_regions(tile, ny, nx):
    assert len(FLAT) == 4
    cpl, rpw, warps, H = tile
    RW, RH, TW = 32 * cpl, rpw * warps, 32 * cpl - 2 * H
    rng = np.random.default_rng(H + nx)
    x, d = rng.standard_normal((2, ny, nx))
    gi, gj = np.arange(nx), np.arange(ny)
    odd = nx % 2 or ny % 2
    assert TW % cpl == 0 and H % cpl == 0
    for red_black in (False, True):
        for k in sorted({1, H // 2 + 1, H}):
            for first in (0, 1) if red_black else (0,):
                want = x
                for s in range(k):
                    mask = parity(gi, gj) == (first + s) % 2 if red_black else True
                    want = half_sweep(want, d, mask, None)
                stored, out = np.zeros((ny, nx), int), np.full((ny, nx), np.nan)
                TH = RH - 2 * k
                for by in range(-(-ny // TH)):
                    for bx in range(-(-nx // TW)):
                        xl, yl = bx * TW - H + np.arange(RW), by * TH - k + np.arange(RH)
                        p, dd = x[np.ix_(yl % ny, xl % nx)], d[np.ix_(yl % ny, xl % nx)]
                        if not odd:  # colours from the region's own indices and its first row's parity
                            colour = (parity(np.arange(RW), np.arange(RH)) + yl[0]) & 1
                        else:
                            colour = parity(xl % nx, yl % ny)
                        for s in range(k):
                            mask = colour == (first + s) % 2 if red_black else True
                            p = half_sweep(p, dd, mask, np.nan)
                        cols = slice(H, min(RW - H, H + nx - bx * TW))
                        rows = slice(k, min(RH - k, k + ny - by * TH))
                        at = np.ix_(yl[rows], xl[cols])
                        stored[at] += 1
                        out[at] = p[rows, cols]
                assert (stored == 1).all()
                np.testing.assert_array_equal(out, want)


# ---------------------------------------------------------- weight gradients
def _plane(pixels, chunks):
    want, b = 16 if chunks >= 8 else 128 // chunks, pixels * 16
    while b % 128 != want:
        b += 16
    return b


WG = [tuple(map(int, t)) for t in re.findall(r"^\s*FS_WG\((\d+), (\d+), (\d+), (\d+), (\d+)\)", _read("fs_guess.cu"), re.M)]


@pytest.mark.parametrize("cfg", WG)
def test_weight_gradient_operands(cfg):
    """Tiles staged into planes of a row and a chunk, read back as MN-major operands."""
    assert len(WG) == 7
    ci, co, TY, PX, NDX = cfg
    KC, OC = ci // 8, co // 8
    XP, GP = _plane(PX + 2, KC), _plane(PX, OC)
    xbytes, gbytes = (TY + 2) * KC * XP, TY * OC * GP
    groups = (TY + 2) * KC
    blocks = -(-groups // 16)
    last = 64 if groups - 16 * (blocks - 1) <= 8 else 128
    assert NDX * blocks * TY * co <= 512  # TMEM columns
    B, H, W = 1, TY + 1, PX + 24  # tiles cut in both directions
    rng = np.random.default_rng(ci + co)
    X = rng.integers(-4, 5, (B, H, W, ci)).astype(np.int64)
    G = rng.integers(-4, 5, (B, H, W, co)).astype(np.int64)
    want = np.zeros((3, 3, ci, co), np.int64)
    for ky in range(3):
        for kx in range(3):
            want[ky, kx] = np.einsum("bhwi,bhwo->io", np.roll(X, (1 - ky, 1 - kx), (1, 2)), G)
    got = np.zeros_like(want)

    # address (in elements of 2 bytes) of row m and pixel k of an operand at byte `start`, planes P apart
    def element(start, P, m, k):
        return (start + (m // 8) * P + (k // 8) * 128 + (k % 8) * 16) // 2 + m % 8

    m = np.arange(128)[:, None]
    k = np.arange(PX)[None, :]
    for y0 in range(0, H, TY):
        for x0 in range(0, W, PX):
            stage = np.full((xbytes + gbytes) // 2, 99, np.int64)
            for r in range(TY + 2):
                for c in range(KC):
                    for px in range(PX + 2):
                        at = ((r * KC + c) * XP + px * 16) // 2
                        stage[at:at + 8] = X[0, (y0 - 1 + r) % H, (x0 - 1 + px) % W, 8 * c:8 * c + 8]
            for r in range(TY):
                for c in range(OC):
                    for px in range(PX):
                        at = (xbytes + (r * OC + c) * GP + px * 16) // 2
                        inside = y0 + r < H and x0 + px < W
                        stage[at:at + 8] = G[0, y0 + r, x0 + px, 8 * c:8 * c + 8] if inside else 0
            b = stage[element(xbytes, GP, np.arange(TY * co)[:, None], k)]
            for dx in range(3):
                for j in range(blocks):
                    rows = last if j == blocks - 1 else 128
                    at = element(dx * 16, XP, 128 * j + m[:rows], k)
                    assert at.max() < stage.size  # rows beyond the tile's stay in the stage
                    D = stage[at] @ b.T
                    for r in range(rows):
                        xrow, c = divmod(128 * j + r, ci)
                        for g in range(TY):
                            if 0 <= xrow - g < 3 and xrow < TY + 2:
                                got[xrow - g, dx, c] += D[r, g * co:(g + 1) * co]
    np.testing.assert_array_equal(got, want)


# ------------------------------------------------------------- convolutions
CONV = [tuple(map(int, t)) for t in re.findall(r"CASE\((\d+), (\d+), (\d+), (\d+), (\d+)\)", _read("fs_conv.cu"))]


@pytest.mark.parametrize("cfg", CONV)
@pytest.mark.parametrize("strips, tiles", [(1, 1), (1, 9), (3, 1), (4, 2), (3, 7)])
def test_convolution_ring(cfg, strips, tiles):
    """Walk and the staging warps' waits: when a tile's rows are copied, the tiles that
    need not be done by then still find theirs in the ring."""
    assert len(CONV) == 7
    _, _, TY, _, D = cfg
    NR = TY * (D + 1) + 2
    order = []  # (strip, first image row, ring row, first of its strip)
    ring = 0
    for s in range(strips):
        for t in range(tiles):
            order.append((s, t * TY, ring, t == 0))
            ring = (ring + (TY if t + 1 < tiles else TY + 2)) % NR
    content = [None] * NR
    done = -1  # the last tile whose MMAs have been waited for
    for k, (s, y, r0, first) in enumerate(order):
        done = max(done, k - 1 if first else k - D - 1)
        for r in range(0 if first else 2, TY + 2):
            content[(r0 + r) % NR] = (s, y - 1 + r)
        for j in range(done + 1, k + 1):
            sj, yj, rj, _ = order[j]
            for r in range(TY + 2):
                assert content[(rj + r) % NR] == (sj, yj - 1 + r), (k, j, r)
