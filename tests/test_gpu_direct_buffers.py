"""Device buffers that the stage calls read and write directly: the results equal those through host buffers bit for
bit, the context keeps its own copies for the next stage, and buffers that share memory or are not on an 8-byte
boundary give the same."""
import numpy as np
import pytest
import torch

from tests.helpers import small_case

pytestmark = pytest.mark.gpu


def _same(a, b):
    return torch.equal(torch.view_as_real(a.cpu()), torch.view_as_real(b.cpu()))


@pytest.mark.parametrize("nxmax,D,c_aber", [(32, 128, 1), (125, 512, 1), (64, 256, 0)])
def test_stage_buffers(nxmax, D, c_aber):
    from mtd_transmission_gb300 import Context, Geometry
    M, N = 5, 150  # a stack of one launch, and of several
    acq, _, d = small_case("plain_512_born", M=M, nxmax=nxmax, dim_final=D, c_aber=c_aber)
    F = 2 * nxmax
    idx = np.arange(N) % M
    with Context(Geometry.from_acquisition(acq), N) as ctx:
        ctx.set_mask(np.ascontiguousarray(d["mask"]))
        for n in (M, N):
            holos = torch.from_numpy(np.ascontiguousarray(d["holos"][idx[:n]]))
            sh = torch.zeros((n, F, F), dtype=torch.complex64)
            fh, ph = torch.zeros_like(sh), torch.zeros(2 * n, dtype=torch.int32)
            vh = torch.zeros((D, D, D))
            ctx.extract(holos, spectra_out=sh)
            ctx.fields(sh, fields_out=fh, posspec_out=ph)
            ctx.reconstruct(fh, ph, indice=vh)
            sd, fd = sh.cuda() * 0, sh.cuda() * 0
            pd, vd = ph.cuda(), torch.zeros((D, D, D), device="cuda")
            torch.cuda.synchronize()
            ctx.extract(holos.cuda(), spectra_out=sd)
            ctx.fields(sd, fields_out=fd, posspec_out=pd)
            ctx.reconstruct(fd, pd, indice=vd)
            ctx.synchronize()
            assert _same(sd, sh) and _same(fd, fh) and torch.equal(vd.cpu(), vh)
            # the context's own copies
            fo, vo = torch.zeros_like(fd), torch.zeros_like(vd)
            torch.cuda.synchronize()
            ctx.fields(None, n=n, fields_out=fo)
            ctx.reconstruct(None, None, n=n, indice=vo)
            ctx.synchronize()
            assert _same(fo, fh) and torch.equal(vo.cpu(), vh)
            # in place, overlapping by half an angle, and 4-byte aligned
            both = torch.zeros(((n + 1) * F * F,), dtype=torch.complex64, device="cuda")
            for shift in (0, F * F // 2):
                src = both[shift:shift + n * F * F].view(n, F, F)
                src.copy_(sd)
                torch.cuda.synchronize()
                out = both[:n * F * F].view(n, F, F)
                ctx.fields(src, fields_out=out)
                ctx.synchronize()
                assert _same(out, fh)
            odd = torch.zeros(2 * n * F * F + 1, device="cuda")
            src = odd[1:].view(n, F, F, 2)
            src.copy_(torch.view_as_real(sd))
            torch.cuda.synchronize()
            out = torch.zeros(2 * n * F * F + 1, device="cuda")[1:].view(n, F, F, 2)
            torch.cuda.synchronize()
            ctx.fields(src, fields_out=out)
            ctx.synchronize()
            assert torch.equal(out.cpu(), torch.view_as_real(fh))
