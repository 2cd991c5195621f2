"""The warp-specialised kernels' stage when the z neighbours' layers come by
bulk copy (ws.cuh), emulated on the CPU from the exported staging tables:

each population plane k lands at its pull shift; the 64-cell layer of the -z
(+z) neighbour lands for the 9 planes with c_z = +1 (-1) beside it; then the
out-of-block values of the other neighbours -- and those of a z neighbour that
is absent -- are written at their table slots.  Every pull of every cell must
then read its own source."""
import ctypes as C

import numpy as np
import pytest

from openludwig_b200 import _native as N

HALO = 3176
ZLO, ZHI = 4, 22


def _c(k):
    return k % 3 - 1, (k // 3) % 3 - 1, k // 9 - 1


@pytest.mark.parametrize("absent", [(), (ZLO,), (ZHI,), (ZLO, ZHI)],
                         ids=["both_z", "no_lower", "no_upper", "no_z"])
def test_stage_with_z_layers_delivers_every_pull(absent):
    sizes = (C.c_int32 * 4)()
    N.call("ol_staging_tables", None, 0, None, 0, sizes)
    w = (C.c_uint32 * sizes[1])()
    N.call("ol_staging_tables", None, 0, w, sizes[1], sizes)
    w, plane, pad = np.array(w, np.int64), sizes[2], sizes[3]
    rng = np.random.default_rng(1)
    blocks = rng.normal(size=(27, 27, 512))        # [neighbour direction][k][cell]
    S = np.full(27 * plane, np.nan)
    for k in range(27):
        cx, cy, cz = _c(k)
        at = k * plane + pad + 8 * cy + 64 * cz
        S[at:at + 512] = blocks[13, k]
    for zdir, cz, layer, off in ((ZLO, 1, slice(448, 512), 0), (ZHI, -1, slice(0, 64), 448)):
        if zdir in absent:
            continue
        for k in range(27):
            if _c(k)[2] != cz:
                continue
            at = k * plane + pad + 8 * _c(k)[1] + off
            assert at % 4 == 0 and k * plane <= at and at + 64 <= (k + 1) * plane
            S[at:at + 64] = blocks[zdir, k, layer]
    inner = 0
    for i in range(HALO):
        k, d, src = int(w[i]) & 31, (int(w[i]) >> 5) & 31, (int(w[i]) >> 10) & 511
        if d in (ZLO, ZHI) and d not in absent:
            continue
        inner += 1
        S[int(w[HALO + 384 + i])] = blocks[d, k, src]
    assert inner == 2208 + 484 * len(absent)
    for k in range(27):
        cx, cy, cz = _c(k)
        for t in range(512):
            x, y, z = t % 8 - cx, (t // 8) % 8 - cy, t // 64 - cz
            d = (x // 8 + 1) + 3 * (y // 8 + 1) + 9 * (z // 8 + 1)
            assert S[k * plane + pad + t - cx] == blocks[d, k, x % 8 + 8 * (y % 8) + 64 * (z % 8)]
