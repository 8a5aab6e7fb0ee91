"""The separable sphere fill's method on the CPU: discs per column and plane,
cut down within the column and by the neighbouring columns, painted as chords,
against the oracle's propagated map (selected and non-selected voxels)."""

import math

import numpy as np
import pytest

import oracle as O


def template2(rmax, off):
    """max |u + off|^2 over 2-D lattice points |u|^2 <= rho, for every rho."""
    t = np.zeros(rmax + 1, np.int64)
    r = math.isqrt(rmax) + 1
    for a in range(r + 1):
        for b in range(r + 1):
            if a * a + b * b <= rmax:
                t[a * a + b * b] = max(t[a * a + b * b], (a + off[0]) ** 2 + (b + off[1]) ** 2)
    return np.maximum.accumulate(t)


def column_list(col, ridge, z):
    """Discs (R, rho) of one column at plane z: outward scan to the first site on each side."""
    out, rcur = [], 0
    for dz in range(len(col)):
        best = 0
        for s in ({z} if dz == 0 else {z - dz, z + dz}):
            lo, hi = min(s, z), max(s, z)
            if 0 <= s < len(col) and all(col[k] for k in range(lo, hi + 1) if k != z) and ridge[s]:
                best = max(best, int(col[s]))
        if best > rcur and best >= dz * dz:
            while out and out[-1][1] <= best - dz * dz:
                out.pop()
            out.append((best, best - dz * dz))
            rcur = best
    return out


def separable_fill(d2, ridge):
    d, h, w = d2.shape
    rmax = int(d2.max())
    face, corner = template2(rmax, (1, 0)), template2(rmax, (1, 1))
    out = np.zeros((d, h, w), np.int64)
    for z in range(d):
        lists = [[column_list(d2[:, y, x], ridge[:, y, x], z) for x in range(w)] for y in range(h)]
        for y in range(h):
            for x in range(w):
                for R, rho in lists[y][x]:
                    def covered(dx, dy, need):
                        yy, xx = y + dy, x + dx
                        return 0 <= yy < h and 0 <= xx < w and any(a >= R and b >= need for a, b in lists[yy][xx])
                    if any(covered(dx, dy, face[rho]) for dx, dy in ((-1, 0), (1, 0), (0, -1), (0, 1))) or \
                       any(covered(dx, dy, corner[rho]) for dx in (-1, 1) for dy in (-1, 1)):
                        continue
                    r = math.isqrt(rho)
                    for yy in range(max(y - r, 0), min(y + r, h - 1) + 1):
                        hw = math.isqrt(rho - (yy - y) ** 2)
                        seg = out[z, yy, max(x - hw, 0):x + hw + 1]
                        np.maximum(seg, R, out=seg)
    return out


def ridge_mask(d2):
    """local_thickness.rs:104-167 with brute-force search templates."""
    rmax = int(d2.max())
    r = math.isqrt(rmax) + 1
    t = np.zeros((4, rmax + 1), np.int64)
    for i in range(r + 1):
        for j in range(r + 1):
            for k in range(r + 1):
                q = i * i + j * j + k * k
                if q <= rmax:
                    for c, o in ((1, (1, 0, 0)), (2, (1, 1, 0)), (3, (1, 1, 1))):
                        t[c, q] = max(t[c, q], (i + o[0]) ** 2 + (j + o[1]) ** 2 + (k + o[2]) ** 2)
    t = np.maximum.accumulate(t, axis=1)
    p = np.pad(d2, 1)
    ridge = d2 > 0
    d, h, w = d2.shape
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                c = abs(dz) + abs(dy) + abs(dx)
                if c:
                    n = p[1 + dz:1 + dz + d, 1 + dy:1 + dy + h, 1 + dx:1 + dx + w]
                    ridge &= ~((d2 > 0) & (n >= t[c][d2]))
    return ridge


@pytest.mark.parametrize("shape,p,seed", [((9, 10, 11), 0.9, 1), ((12, 9, 14), 0.97, 2), ((15, 8, 9), 0.6, 3),
                                          ((16, 16, 16), 0.995, 4), ((2, 7, 12), 0.9, 5)])
@pytest.mark.parametrize("phase", [0, 1])
def test_separable_fill_matches_the_propagated_map(shape, p, seed, phase):
    vol = (np.random.default_rng(seed).random(shape) < p).astype(np.uint8)
    if phase:
        vol = 1 - vol
    ref = O.local_thickness(vol, phase)
    d2 = ref.edt.astype(np.int64).reshape(shape)
    assert np.array_equal(separable_fill(d2, ridge_mask(d2)), ref.propagated.astype(np.int64))
