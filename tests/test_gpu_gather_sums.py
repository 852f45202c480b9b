"""Cap sums where every lane of a group hits the same planes: a stack whose angles all share one or two specular
positions, with values over six decades and both signs, scattered by the adjoint and normalised by the
reconstruction, against the oracle."""
import numpy as np
import pytest

import oracle
from tests.helpers import oracle_cfg, rel_l2, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,spread", [(1, 0), (32, 0), (70, 0), (70, 1), (1100, 1)])
def test_shared_planes(M, spread):
    from mtd_transmission_gb300 import Context, Geometry
    acq, _, _ = small_case(M=1, ccd_roix=256, nxmax=32, circle_cx=64, circle_cy=64, dim_final=128)
    F, D = 64, 128
    r = np.random.default_rng(M + spread)
    caps = (10.0 ** r.uniform(-3, 3, (M, F, F)) * np.exp(2j * np.pi * r.random((M, F, F)))).astype(np.complex64)
    p = np.full((M, 2), 32) + spread * np.arange(M)[:, None] % 2 * np.array([7, -4])
    pos = np.ascontiguousarray(p.T.reshape(-1).astype(np.int32))
    cfg, pf = oracle_cfg(acq), p.T.reshape(-1).astype(np.float64)
    with Context(Geometry.from_acquisition(acq), M) as ctx:
        an, ak = ctx.adjoint(caps, n=M, posspec=pos, absorption_out=np.zeros((D, D, D), np.float32))
        cnt, re = np.zeros((D, D, D), np.uint32), np.zeros((D, D, D), np.float32)
        ctx.reconstruct(caps, pos, indice=re, counts=cnt)
    ref = oracle.adjoint_caps(caps.astype(np.complex128), pf, cfg)
    # the sums' own rounding (2^-24 of each cell's sum, whose terms may cancel) and the FP32 transform's
    assert rel_l2(an, ref.real) <= 2e-6 and rel_l2(ak, ref.imag) <= 2e-6
    ref = oracle.reconstruction(caps.astype(np.complex128), pf, cfg)
    assert np.array_equal(cnt, ref["counts"].astype(np.uint32))
    assert rel_l2(re, ref["indice"].real) <= 1e-5
