"""The bound of the density pass's candidate filter (csrc/sph.cu, tile_neighbors)
on the weakest arithmetic that the PTX specification allows its contraction:
products and sums of the accumulators' precision in any order and rounding,
subnormal operands kept or taken as zero. A pair inside the support is marked
by it, wherever the pair lies in its group. CPU only."""

from __future__ import annotations

import re
from pathlib import Path

import numpy as np
import pytest

SOURCE = (Path(__file__).resolve().parents[1] / "newton_sph_dev_b200" / "csrc" / "sph.cu").read_text()
F = np.float32


def _filter():
    """The accumulators' type, and the two expressions of the filter's bound."""
    acc = re.search(r"mma\.sync\.aligned\.m16n8k8\.row\.col\.(f\d+)\.f16\.f16\.(f\d+) ", SOURCE)
    d, thr = (re.search(rf"const float {name} = ([^;]*);", SOURCE) for name in ("d", "thr"))
    assert acc and d and thr and acc[1] == acc[2]
    plain = lambda m: re.sub(r"([0-9.]+(?:e-?\d+)?)f\b", r"F(\1)", m[1]).replace("sqrtf", "np.sqrt")  # noqa: E731
    return {"f16": np.float16, "f32": np.float32}[acc[1]], plain(d), plain(thr)


def _half(a):
    return a.astype(np.float16).astype(F)


def _up(exact, kind):
    """`exact` (64 bits) rounded towards plus infinity to `kind`."""
    low = exact.astype(kind)
    return np.where(low.astype(np.float64) < exact, np.nextafter(low, kind(np.inf)), low).astype(np.float64)


def _pairs(rng, n, span, cells, offset):
    """Particles a of groups `span` supports long in x and about `cells` wide in
    y and z, and b of each at h (1 - 2^-22), in units of h around the group's
    origin; the group's largest coordinates."""
    a = np.stack([rng.uniform(-span / 2, span / 2, n), rng.uniform(-cells, cells, n), rng.uniform(-cells, cells, n)], 1)
    a[: n // 4, 0] = np.where(rng.random(n // 4) < 0.5, span / 2, -span / 2)
    a[: n // 8, 1:] = np.where(rng.random((n // 8, 2)) < 0.5, cells, -cells)
    e = rng.normal(size=(n, 3))
    e[::5] *= [1, 0, 0]
    e[1::5] = np.sign(a[1::5])  # outwards
    e /= np.linalg.norm(e, axis=1)[:, None]
    b = a + e * (1 - 2.0**-22)
    a[3::7, 1], b[4::7, 2] = 3e-5, -2e-5  # subnormal in 16 bits
    far = ((a - b) ** 2).sum(1) >= (1 - 2.0**-23) ** 2
    b[far] = a[far] + e[far] * (1 - 2.0**-22)
    return (a + offset).astype(F), (b + offset).astype(F), F(offset)


@pytest.mark.parametrize("flush", [False, True])
@pytest.mark.parametrize("span,cells", [(0.1, 0.3), (4.0, 0.3), (12.0, 1.0), (30.0, 2.5), (48.0, 4.0), (100.0, 8.0)])
def test_no_neighbour_is_missed(span, cells, flush):
    acc, d_of, thr_of = _filter()
    rng = np.random.default_rng(int(10 * span))
    a, b, origin = _pairs(rng, 40000, span, cells, 17.0)
    u, w = (a - origin).astype(F), (b - origin).astype(F)  # (inv_h = 1)
    mx = F(np.abs(u[:, 0]).max()) + F(1.01)
    myz = F(np.abs(u[:, 1:]).max()) + F(1.01)
    big = mx * mx + F(2) * myz * myz
    if not big < 4096:
        return  # the kernel leaves such a group to the general scan
    known = dict(F=F, np=np, mx=mx, myz=myz, big=big)
    known["d"] = eval(d_of, known)
    thr = eval(thr_of, known)
    assert thr.dtype == F and 1 < thr < 2
    hu, hw = _half(u), _half(w)
    norm = lambda h: (h[:, 2] * h[:, 2] + (h[:, 1] * h[:, 1] + h[:, 0] * h[:, 0])).astype(F)  # noqa: E731
    na, nb = norm(hu) - thr, norm(hw)
    ah, bh = _half(na), _half(nb)
    one = np.ones(len(u), F)
    left = np.stack([-2 * hu[:, 0], -2 * hu[:, 1], -2 * hu[:, 2], one, one, ah, _half(na - ah)], 1)
    right = np.stack([hw[:, 0], hw[:, 1], hw[:, 2], bh, _half(nb - bh), one, one], 1)
    if flush:
        left, right = (np.where(np.abs(m) < 2.0**-14, F(0), m) for m in (left, right))
    products = _up(left.astype(np.float64) * right.astype(np.float64), acc)
    order = np.argsort(products, 1)
    for o in (order, order[:, ::-1], np.argsort(-np.abs(products), 1), np.argsort(rng.random(products.shape), 1)):
        p = np.take_along_axis(products, o, 1)
        total = np.zeros(len(p))
        for k in range(p.shape[1]):
            total = _up(total + p[:, k], acc)
        inside = ((a.astype(np.float64) - b.astype(np.float64)) ** 2).sum(1) < 1
        missed = inside & ~(total < 0)
        assert inside.sum() > 10000 and not missed.any(), f"{missed.sum()} of {inside.sum()} pairs lost"
