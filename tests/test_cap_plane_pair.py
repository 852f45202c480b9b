"""The cap plane's decision near rounding boundaries from pairs of floats, against FP64 (CPU).

Where the float heights' difference comes within 1e-3 of a rounding boundary, cap_plane decides by the heights as
pairs of floats (nearest float and remainder) unless that difference comes within 1e-8 of the boundary.  numpy's
float32 arithmetic rounds as the kernel's does; for every such bin of the checked angles the decision must be the
FP64 rounding, and nearly none may be left to FP64."""
import numpy as np
import pytest

from mtd_transmission_gb300 import Geometry, api
from tests import simul

F32 = np.float32


@pytest.mark.parametrize("name", ["plain_512_born", "rytov_1024", "tomo_config_1024", "large_2048"])
def test_pair_decision(name):
    acq, _, _ = simul.workload(name)
    r2 = int(api.derive(Geometry.from_acquisition(acq))["rayon"] ** 2)
    N = acq.nxmax
    fd = np.arange(-N, N)
    d2 = (fd[:, None] ** 2 + fd[None, :] ** 2).ravel()
    s64 = np.sqrt((r2 - np.unique(d2[d2 < N * N])).astype(np.float64))
    hi = s64.astype(F32)
    lo = (s64 - hi).astype(F32)
    r = np.random.default_rng(3)
    near = left = 0
    for tx, ty in r.integers(-int(0.65 * N), int(0.65 * N) + 1, (400, 2)):
        f64 = np.sqrt(np.float64(r2 - tx * tx - ty * ty))
        fh = F32(f64)
        fl = F32(f64 - fh)
        d = hi - fh
        below = np.floor(d)
        m = np.abs((d - below) - F32(0.5)) <= F32(1e-3)
        a, al, d, below, ref = hi[m], lo[m], d[m], below[m], s64[m] - f64
        v = d - a
        e = (a - (d - v)) - (fh + v)
        t = (d - (below + F32(0.5))) + (e + (al - fl))
        assert t.dtype == F32
        sure = np.abs(t) > F32(1e-8)
        want = np.sign(ref) * np.floor(np.abs(ref) + 0.5)
        got = np.where(t > 0, below + 1, below)
        assert np.array_equal(got[sure], want[sure]), (tx, ty)
        assert np.abs(t.astype(np.float64) - (ref - (below.astype(np.float64) + 0.5))).max(initial=0) < 1e-9
        near += m.sum()
        left += (~sure).sum()
    assert near > 100 and left <= 1e-4 * near
