"""The volume stage where caps reach only part of the volume's columns (DIM_FINAL above 4 NXMAX) and where the
window's edge is not a multiple of the kernels' column blocks: every output, to device and to host buffers, against
the oracle, and the operators on the same geometry."""
import numpy as np
import pytest
import torch

import oracle
from tests.helpers import oracle_cfg, rel_l2, small_case

pytestmark = pytest.mark.gpu


def _stack(nxmax, D, M):
    acq, _, _ = small_case(M=1, ccd_roix=512, nxmax=nxmax, dim_final=D)
    F = 2 * nxmax
    r = np.random.default_rng(nxmax)
    fields = (r.standard_normal((M, F, F)) + 1j * r.standard_normal((M, F, F))).astype(np.complex64)
    # the corners of what tilts reach, the centre, and the rest at random
    e = int(0.65 * nxmax)
    p = np.array([[nxmax, nxmax], [nxmax - e, nxmax + e], [nxmax + e, nxmax - e]] +
                 (nxmax + r.integers(-e, e + 1, (M - 3, 2))).tolist())
    return acq, fields, p


@pytest.mark.parametrize("nxmax,D,M", [(32, 256, 40), (32, 128, 3), (125, 512, 3)])
def test_volume_outputs(nxmax, D, M):
    from mtd_transmission_gb300 import Context, Geometry
    acq, fields, p = _stack(nxmax, D, M)
    pos = np.ascontiguousarray(p.T.reshape(-1).astype(np.int32))
    ref = oracle.reconstruction(fields.astype(np.complex128), p.T.reshape(-1).astype(np.float64), oracle_cfg(acq))
    with Context(Geometry.from_acquisition(acq), M) as ctx:
        for dev in ("cuda", "cpu"):
            out = [torch.full((D, D, D), 7, dtype=t, device=dev)
                   for t in (torch.float32, torch.float32, torch.uint8, torch.int32)]
            ctx.reconstruct(fields, pos, indice=out[0], absorption=out[1], otf=out[2], counts=out[3])
            ctx.synchronize()
            re, im, otf, cnt = (o.cpu().numpy() for o in out)
            assert np.array_equal(cnt, ref["counts"].astype(np.int32))
            assert np.array_equal(otf, ref["otf"].astype(np.uint8))
            assert rel_l2(re, ref["indice"].real) <= 1e-5
            assert rel_l2(im, ref["indice"].imag) <= 1e-5


def test_operators_beyond_the_window():
    from mtd_transmission_gb300 import Context, Geometry
    acq, caps, p = _stack(32, 256, 5)
    D, M = 256, 5
    pos = np.ascontiguousarray(p.T.reshape(-1).astype(np.int32))
    r = np.random.default_rng(1)
    x = [r.standard_normal((D, D, D)).astype(np.float32) for _ in range(2)]
    cfg, pf = oracle_cfg(acq), p.T.reshape(-1).astype(np.float64)
    with Context(Geometry.from_acquisition(acq), M) as ctx:
        f = ctx.forward(x[0], x[1], n=M, posspec=pos)
        an, ak = ctx.adjoint(caps, n=M, posspec=pos, absorption_out=np.zeros((D, D, D), np.float32))
    assert rel_l2(f, oracle.forward_caps(x[0].astype(np.float64), x[1].astype(np.float64), pf, cfg)) <= 1e-5
    ref = oracle.adjoint_caps(caps.astype(np.complex128), pf, cfg)
    assert rel_l2(an, ref.real) <= 1e-5 and rel_l2(ak, ref.imag) <= 1e-5
