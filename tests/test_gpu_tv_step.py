"""The projected-gradient step's total-variation term against numpy in FP64: one iteration with a zero data
step, so that x <- clamp(x - tv dTV(x)), at the smallest and a larger volume, with and without the absorption."""
import numpy as np
import pytest

from tests.helpers import small_case

pytestmark = pytest.mark.gpu


def _tv_grad(x, eps):
    g = [np.diff(x, axis=a, append=np.take(x, [-1], axis=a)) for a in range(3)]
    inv = 1.0 / np.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2 + eps ** 2)
    out = -(g[0] + g[1] + g[2]) * inv
    for a in range(3):
        p = g[a] * inv
        sl = [slice(None)] * 3
        sl[a] = slice(1, None)
        sr = [slice(None)] * 3
        sr[a] = slice(None, -1)
        out[tuple(sl)] += p[tuple(sr)]
    return out


@pytest.mark.parametrize("D,nxmax,absn", [(128, 32, True), (128, 32, False), (256, 64, True)])
def test_tv_step(D, nxmax, absn):
    from mtd_transmission_gb300 import Context, Geometry
    acq, _, _ = small_case(M=1, nxmax=nxmax, dim_final=D)
    F = 2 * nxmax
    r = np.random.default_rng(7)
    x = [(0.12 * r.random((D, D, D)) - 0.01).astype(np.float32) for _ in range(2)]
    eps, weight, hi = 2e-3, 5e-2, (0.1, 0.08)
    io = [v.copy() for v in x]
    with Context(Geometry.from_acquisition(acq), 1) as ctx:
        ctx.tv_reconstruct(io[0], io[1] if absn else None, caps=np.zeros((1, F, F), np.complex64),
                           posspec=np.array([nxmax, nxmax], np.int32), iterations=1, init=0, step=0.0,
                           tv_weight=weight, tv_eps=eps, index_max=hi[0], absorption_max=hi[1])
    for c in range(2 if absn else 1):
        tv = np.float64(np.float32(np.float32(weight) * np.float32(hi[c])))
        want = np.clip(x[c] - tv * _tv_grad(x[c].astype(np.float64), np.float64(np.float32(eps))), 0.0,
                       np.float64(np.float32(hi[c])))
        # four terms of magnitude at most sqrt(3), each within a few FP32 roundings (rsqrt 2 ulp), and x's own
        assert np.abs(io[c] - want).max() <= 4e-6 * tv + 1.5e-8
