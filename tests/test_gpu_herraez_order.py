"""Herraez group merging where the order of the merges is hardest to keep: a flat phase (every interior edge of
equal reliability, so the merges run along the rows), noise (residues everywhere), and a phase with a large flat
part.  The unwrapped phase equals the oracle's, bit for bit, on the GPU's own wrapped phase."""
import numpy as np
import pytest

import oracle
from mtd_transmission_gb300 import Context, Geometry
from tests.helpers import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxmax", [32, 125, 128])
@pytest.mark.parametrize("kind", ["flat", "noise", "half"])
def test_merge_order(nxmax, kind):
    M = 2
    acq, _, _ = small_case("rytov_1024", M=M, volkov=0, ccd_roix=512, nxmax=nxmax, circle_cx=128, circle_cy=128,
                           dim_final=512 if nxmax > 64 else 128)
    F = 2 * nxmax
    r = np.random.default_rng(11)
    field = np.ones((M, F, F), np.complex128)
    if kind != "flat":
        noise = np.exp(2j * np.pi * r.random((M, F, F)))
        field = noise if kind == "noise" else np.where(np.arange(F) < F // 2, 4.0, noise)
    spec = np.fft.fft2(field).astype(np.complex64)
    ph, un, fo = (np.zeros((M, F, F), t) for t in (np.float32, np.float32, np.complex64))
    with Context(Geometry.from_acquisition(acq), M) as ctx:
        ctx.fields_debug(spec, fields_out=fo, phase=ph, unwrapped=un)
    for a in range(M):
        ref, _ = oracle.herraez(ph[a].astype(np.float64), a)
        np.testing.assert_array_equal(un[a], ref.astype(np.float32), err_msg=f"angle {a}")
