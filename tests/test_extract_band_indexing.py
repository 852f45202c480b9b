"""Index arithmetic of the extraction's two passes, on the CPU.

The row pass stores the crop's kx band row by row, inter[y][c]; the column
pass's lanes run across the band's columns (16 a CTA, or 8 from 32 lanes a
transform on), load rows j + T n1, and store the crop rows of the output bins
j + q T + E k2, skipping blocks of GR output groups that the crop does not
meet.  This restates that arithmetic for every hologram size, band width (250
leaves the last CTA partly empty) and several crop corners: every band value
is written once and read once, every crop value stored once, no block with a
crop row is skipped, the exchange positions stay inside a transform's array, and
the specular search's partial records and the shared memory fit their limits."""
from __future__ import annotations

import numpy as np
import pytest

ARG_PARTS_MAX = 512


def _warp_fft(H):
    E = 64 if H >= 2048 else 32 if H >= 512 else 16
    return E, H // E, 32 // (H // E)  # points per lane, lanes, transforms per warp


@pytest.mark.parametrize("H", [256, 512, 1024, 2048])
@pytest.mark.parametrize("F", [64, 128, 250, 256, 512])
def test_band_and_crop(H, F):
    if F > H:
        pytest.skip("the crop lies inside the hologram's spectrum")
    E, T, G = _warp_fft(H)
    P, length = 8 * G, H + E  # row pairs per CTA; padded transform length
    stride = length + 1
    pad = lambda i: i + i // T
    assert P * stride * 8 + 8 * 8 <= 227 * 1024  # the barriers of the staged rows are static

    # row pass: every band value once
    seen = np.zeros((H, F), int)
    for bx in range(H // (2 * P)):
        for tr in range(P):
            ya = 2 * (bx * P + tr)
            for j in range(T):
                c = np.arange(j, F, T)
                seen[ya, c] += 1
                seen[ya + 1, c] += 1
    assert (seen == 1).all()
    for x0 in {0, min(1, H - F), (H - F) // 2, H - F}:
        k = x0 + np.arange(F)
        assert pad(k).max() < length and pad((H - k) & (H - 1)).max() < length

    # column pass
    B = 8 if T >= 32 else 16
    NT, grid = B * T, (F + B - 1) // B
    assert B * stride * 8 <= 227 * 1024 and NT <= 1024
    assert grid * (NT // 32) <= ARG_PARTS_MAX
    tid = np.arange(NT)
    t, j = tid % B, tid // B
    c = np.arange(grid)[:, None] * B + t
    valid = c < F
    read = np.zeros((H, F), int)
    for n1 in range(E):
        np.add.at(read, (np.broadcast_to(j + n1 * T, c.shape)[valid], c[valid]), 1)
    assert (read == 1).all()
    GR = 4 if E >= 32 else 2
    assert T % GR == 0 and E % T == 0  # whole groups of output blocks
    for y0 in {min(y, H - F) for y in (0, 1, E - 1, E * GR, (H - F) // 2, (H - F) // 2 + 5, H - F)}:
        stored = np.zeros((F, F), int)
        for g in range(T // GR):
            if E * GR * (g + 1) <= y0 or E * GR * g >= y0 + F:
                continue
            for kk in range(GR):
                for q in range(E // T):
                    r = np.broadcast_to(j + q * T + E * (g * GR + kk) - y0, c.shape)
                    m = valid & (r >= 0) & (r < F)
                    np.add.at(stored, (r[m], c[m]), 1)
        assert (stored == 1).all(), y0
