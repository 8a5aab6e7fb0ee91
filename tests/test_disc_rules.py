"""The rules by which disc_list_kernel leaves discs and rows out, on the CPU: its
cuts against their definition (the kernel's own functions, compiled here), and a
restatement of the rest -- a column's planes cut at its two neighbours, the
largest (rho, R) per cell, the seven cells that may cover a disc, rows cut at
y -+ 1, nothing seen beyond the patch -- against the oracle's propagated map, on
every pattern of a tiny volume and on plateaus of equal radii."""

import itertools
import math
import subprocess

import numpy as np
import pytest

import oracle as O
from bone_morphometry_gb300 import build
from test_disc_math import ridge_mask, template2

PROGRAM = r"""
#include <cstdio>
#include "disc_cuts.h"
int main() {
  for (int gain = -600; gain <= 600; ++gain)
    printf("%d %d %d %d\n", gain, bm::cut_above(gain, true), bm::cut_above(gain, false), bm::cut_below(gain));
}
"""


def cut_above(gain, larger):
    return -((gain - 1) >> 1) - 1 if larger else (1 - gain) >> 1


def cut_below(gain):
    return (gain + 1) >> 1


def test_cuts_are_their_definition(tmp_path):
    src = tmp_path / "cuts.cu"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "cuts")
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, str(src), "-o", exe], check=True)
    lines = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]
    assert len(lines) == 1201
    reach = range(-700, 701)
    for line in lines:
        gain, above_larger, above_equal, below = map(int, line.split())
        # rho - t^2 against rho + gain - (t - 1)^2, one step up; (t + 1)^2, one step down
        assert above_larger == max(t for t in reach if not gain >= 1 - 2 * t)
        assert above_equal == max(t for t in reach if not gain > 1 - 2 * t)
        assert below == min(t for t in reach if not gain >= 1 + 2 * t)
        assert (above_larger, above_equal, below) == (cut_above(gain, True), cut_above(gain, False), cut_below(gain))


def listed_discs(d2, ridge, patch):
    """{plane: [(R, rho, y, x, first row, last row)]} as the kernel lists them; patch: its (rows, columns)."""
    d, h, w = d2.shape
    rmax = int(d2.max())
    face, corner = template2(rmax, (1, 0)), template2(rmax, (1, 1))
    table = np.zeros((d, h, w, 2), np.int64)  # largest (rho, R), rho first
    discs = []
    for z, y, x in zip(*np.nonzero(ridge)):
        R = int(d2[z, y, x])
        rad = math.isqrt(R)
        up = (int(d2[z + 1, y, x]) if z + 1 < d else 0) - R
        dn = (int(d2[z - 1, y, x]) if z > 0 else 0) - R
        hi = min(rad, cut_above(up, up > 0)) if up >= 0 else rad
        lo = max(-rad, cut_below(dn)) if dn >= 0 else -rad
        for t in range(max(lo, -z), min(hi, d - 1 - z) + 1):
            rho = R - t * t
            discs.append((z + t, y, x, R, rho))
            if (rho, R) > tuple(table[z + t, y, x]):
                table[z + t, y, x] = rho, R

    def cell(z, y, x, dy, dx):
        yy, xx = y + dy, x + dx
        if not (0 <= yy < h and 0 <= xx < w) or yy // patch[0] != y // patch[0] or xx // patch[1] != x // patch[1]:
            return 0, 0
        return int(table[z, yy, xx, 0]), int(table[z, yy, xx, 1])

    out = {}
    for z, y, x, R, rho in discs:
        def covers(c, need):
            return c[1] >= R and c[0] >= need
        own = cell(z, y, x, 0, 0)
        if own != (rho, R) and covers(own, rho):
            continue
        if any(covers(cell(z, y, x, 0, dx), face[rho]) for dx in (-1, 1)):
            continue
        if any(covers(cell(z, y, x, dy, dx), corner[rho]) for dy in (-1, 1) for dx in (-1, 1)):
            continue
        half = math.isqrt(rho)
        a, b = cell(z, y, x, 1, 0), cell(z, y, x, -1, 0)
        last = min(half, cut_above(a[0] - rho, a[1] > R)) if a[1] >= R else half
        first = max(-half, cut_below(b[0] - rho)) if b[1] >= R else -half
        if first <= last:
            out.setdefault(z, []).append((R, rho, y, x, first, last))
    return out


def painted(d2, ridge, patch):
    d, h, w = d2.shape
    out = np.zeros((d, h, w), np.int64)
    for z, discs in listed_discs(d2, ridge, patch).items():
        for R, rho, y, x, first, last in discs:
            for t in range(max(first, -y), min(last, h - 1 - y) + 1):
                half = math.isqrt(rho - t * t)
                seg = out[z, y + t, max(x - half, 0):x + half + 1]
                np.maximum(seg, R, out=seg)
    return out


def assert_rules(vol, patches):
    ref = O.local_thickness(vol, 0)
    d2 = ref.edt.astype(np.int64).reshape(vol.shape)
    ridge = ridge_mask(d2)
    for patch in patches:
        assert np.array_equal(painted(d2, ridge, patch), ref.propagated.astype(np.int64).reshape(vol.shape)), patch


WHOLE = (1 << 20, 1 << 20)


@pytest.mark.parametrize("shape", [(2, 2, 3), (2, 3, 2), (3, 2, 2)])
def test_every_pattern_of_a_tiny_volume(shape):
    n = math.prod(shape)
    for bits in itertools.product((0, 1), repeat=n):
        if 0 < sum(bits) < n:
            assert_rules(np.array(bits, np.uint8).reshape(shape), [WHOLE])


def slab(shape, axis, at):
    """All selected but planes across an axis: every ridge voxel between two of them has the same radius."""
    vol = np.ones(shape, np.uint8)
    index = [slice(None)] * 3
    for k in at:
        index[axis] = k
        vol[tuple(index)] = 0
    return vol


PLATEAUS = [("slab-%s-%d" % ("zyx"[axis], gap), slab((13, 12, 14), axis, (0, gap))) for axis in range(3) for gap in (5, 6, 11)]
PLATEAUS += [("one-plane-" + "zyx"[axis], slab((9, 8, 10), axis, (3,))) for axis in range(3)]


def bars(shape, step):
    """Selected bars of a square section along x: plateaus along a line."""
    vol = np.ones(shape, np.uint8)
    vol[::step] = 0
    vol[:, ::step] = 0
    return vol


PLATEAUS += [("bars-%d" % s, bars((13, 13, 9), s)) for s in (4, 5)]
PLATEAUS += [("bars-z-%d" % s, np.ascontiguousarray(bars((13, 13, 9), s).transpose(2, 1, 0))) for s in (4, 5)]


def corners():
    vol = np.ones((9, 9, 9), np.uint8)
    vol[::8, ::8, ::8] = 0
    return vol


def chequer():
    z, y, x = np.indices((8, 9, 10)) // 2
    return ((z + y + x) % 2).astype(np.uint8)


PLATEAUS += [("corners", corners()), ("chequer", chequer())]


@pytest.mark.parametrize("name,vol", PLATEAUS, ids=[p[0] for p in PLATEAUS])
def test_plateaus_of_equal_radii(name, vol):
    assert_rules(vol, [WHOLE, (8, 32), (3, 4)])


@pytest.mark.parametrize("shape,p,seed", [((9, 10, 11), 0.9, 1), ((12, 9, 14), 0.97, 2), ((15, 8, 9), 0.6, 3),
                                          ((16, 16, 16), 0.995, 4), ((2, 7, 12), 0.9, 5), ((6, 18, 40), 0.97, 6)])
def test_random_volumes(shape, p, seed):
    assert_rules((np.random.default_rng(seed).random(shape) < p).astype(np.uint8), [WHOLE, (8, 32), (2, 3)])
