"""Intermediates that the caller wants stored over the spectra they come from, for a stack of more angles than one
launch takes: the spectra of the later launches are still unread when the first one's results are stored."""
import numpy as np
import pytest

from tests.helpers import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["phase", "unwrapped", "amp"])
def test_debug_output_over_spectra(which):
    import torch
    from mtd_transmission_gb300 import Context, Geometry
    acq, _, _ = small_case(M=1, ccd_roix=256, nxmax=32, circle_cx=64, circle_cy=64, dim_final=128)
    n, F = 130, 64  # two launches of 65
    gen = torch.Generator(device="cuda").manual_seed(3)
    spectra = 0.02 * torch.randn((n, F, F), generator=gen, device="cuda", dtype=torch.complex64)
    spectra[:, 20, 30] = 50.0
    apart, fields, want = torch.zeros((n, F, F), device="cuda"), torch.zeros_like(spectra), torch.zeros_like(spectra)
    both = spectra.clone()
    half = torch.view_as_real(both).reshape(2, n, F, F)[1]  # the second half of the spectra's memory, as floats
    torch.cuda.synchronize()
    with Context(Geometry.from_acquisition(acq), n) as ctx:
        ctx.fields_debug(spectra, fields_out=want, **{which: apart})
        ctx.fields_debug(both, fields_out=fields, **{which: half})
    assert torch.equal(half, apart) and torch.equal(fields, want)
