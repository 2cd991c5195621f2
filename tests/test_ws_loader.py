"""The warp-specialised kernels' loads (ws.cuh), emulated on the CPU from the
loader table as the kernels read it (ol_ws_loader_sources runs their own index
functions on the host):

* the table holds every out-of-block pull once, those of the z face neighbours
  last, and each entry's source is k * dstride + neighbour + cell, also where
  the 27 planes reach beyond 32-bit element offsets;
* the stage when the z neighbours' layers come by bulk copy: each population
  plane k lands at its pull shift; the 64-cell layer of the -z (+z) neighbour
  lands for the 9 planes with c_z = +1 (-1) beside it; then the out-of-block
  values of the other neighbours -- and those of a z neighbour that is absent --
  are written at their table slots.  Every pull of every cell must then read its
  own source."""
import ctypes as C

import numpy as np
import pytest

from openludwig_b200 import _native as N

HALO, INNER = 3176, 2208
ZLO, ZHI = 4, 22


def _c(k):
    return k % 3 - 1, (k // 3) % 3 - 1, k // 9 - 1


def _staging():
    sizes = (C.c_int32 * 4)()
    N.call("ol_staging_tables", None, 0, None, 0, sizes)
    w = (C.c_uint32 * sizes[1])()
    N.call("ol_staging_tables", None, 0, w, sizes[1], sizes)
    return np.array(w, np.int64), sizes[2], sizes[3]


def _loader(dstride, neighbours):
    n = C.c_int32()
    rows = np.zeros((HALO, 4), np.int64)
    nb = np.ascontiguousarray(neighbours, np.int32)
    N.call("ol_ws_loader_sources", C.c_int64(dstride), nb.ctypes.data, rows.ctypes.data, HALO,
           C.byref(n))
    assert n.value == HALO
    return rows


# 512-cell multiples; 27 planes of 159 072 862 elements end just below 2^32
@pytest.mark.parametrize("dstride", [27 * 512, 512 * 4096, 159_072_768, 159_073_280, 400_000_000,
                                     2 ** 31 - 512], ids=str)
def test_loader_sources(dstride):
    w, plane, pad = _staging()
    blocks = dstride // 512
    rng = np.random.default_rng(3)
    for trial in range(3):
        nb = 512 * rng.integers(0, blocks, 27)
        if trial == 0:
            nb[:] = 512 * (blocks - 1)          # the largest offsets
        absent = rng.random(27) < 0.3 if trial == 2 else np.zeros(27, bool)
        rows = _loader(dstride, np.where(absent, -1, nb))
        assert sorted(rows[:, 3]) == list(range(HALO))
        e = w[rows[:, 3]]
        k, d, src, cell = e & 31, (e >> 5) & 31, (e >> 10) & 511, e >> 19
        assert np.array_equal(rows[:, 2], d)
        assert np.array_equal(rows[:, 0], np.where(absent[d], -1, k * dstride + nb[d] + src))
        assert np.array_equal(rows[:, 1], k * plane + pad + cell - (k % 3 - 1))
        assert not np.isin(d[:INNER], (ZLO, ZHI)).any()
        half = (HALO - INNER) // 2
        assert (d[INNER:INNER + half] == ZLO).all() and (d[INNER + half:] == ZHI).all()


@pytest.mark.parametrize("absent", [(), (ZLO,), (ZHI,), (ZLO, ZHI)],
                         ids=["both_z", "no_lower", "no_upper", "no_z"])
def test_stage_with_z_layers_delivers_every_pull(absent):
    _, plane, pad = _staging()
    dstride = 27 * 512
    rows = _loader(dstride, 512 * np.arange(27))   # neighbour d is block d, block 13 the own one
    rng = np.random.default_rng(1)
    f = rng.normal(size=(27, dstride))             # [k][block, cell]
    S = np.full(27 * plane, np.nan)
    for k in range(27):
        at = k * plane + pad + 8 * _c(k)[1] + 64 * _c(k)[2]
        S[at:at + 512] = f[k, 13 * 512:14 * 512]
    for zdir, cz, layer, off in ((ZLO, 1, 448, 0), (ZHI, -1, 0, 448)):
        if zdir in absent:
            continue
        for k in range(27):
            if _c(k)[2] != cz:
                continue
            at = k * plane + pad + 8 * _c(k)[1] + off
            assert at % 4 == 0 and k * plane <= at and at + 64 <= (k + 1) * plane
            S[at:at + 64] = f[k, zdir * 512 + layer:zdir * 512 + layer + 64]
    half = (HALO - INNER) // 2
    carried = list(range(INNER))
    carried += range(INNER, INNER + half) if ZLO in absent else []
    carried += range(INNER + half, HALO) if ZHI in absent else []
    for offset, slot, _, _ in rows[carried]:
        S[slot] = f.reshape(-1)[offset]
    for k in range(27):
        cx, cy, cz = _c(k)
        for t in range(512):
            x, y, z = t % 8 - cx, (t // 8) % 8 - cy, t // 64 - cz
            d = (x // 8 + 1) + 3 * (y // 8 + 1) + 9 * (z // 8 + 1)
            assert S[k * plane + pad + t - cx] == f[k, d * 512 + x % 8 + 8 * (y % 8) + 64 * (z % 8)]
