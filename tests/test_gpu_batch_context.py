"""A context that a batch was captured from goes on working by itself: every entry point after the batch's creation,
after its launches and after its end, with the results of a context that was never captured."""
import numpy as np
import pytest

from tests.helpers import small_case

pytestmark = pytest.mark.gpu


def test_calls_around_a_batch():
    import torch
    from mtd_transmission_gb300 import Batch, Context, Geometry
    acq, _, d = small_case("plain_512_born", M=20)
    D, F = acq.dim_final, acq.F
    holos = torch.from_numpy(np.ascontiguousarray(d["holos"])).cuda()
    vol = lambda: torch.zeros((D, D, D), device="cuda")

    def calls(ctx):
        out = [vol(), vol(), torch.zeros((20, F, F), dtype=torch.complex64, device="cuda"),
               torch.zeros((20, F, F), dtype=torch.complex64, device="cuda"), vol(), vol(), vol()]
        torch.cuda.synchronize()
        for re in (out[0], out[5]):  # both of a context's record buffers
            ctx.pipeline(holos, indice=re, absorption=out[1])
        ctx.extract(holos, spectra_out=out[2])
        ctx.fields(out[2], fields_out=out[3])
        ctx.reconstruct(n=20, indice=out[4])
        ctx.adjoint(out[3], n=20, index_out=out[6])
        ctx.synchronize()
        return out

    with Context(Geometry.from_acquisition(acq), 20) as alone, Context(Geometry.from_acquisition(acq), 20) as ctx:
        for c in (alone, ctx):
            c.set_mask(np.ascontiguousarray(d["mask"]))
        want = calls(alone)
        re, im = vol(), vol()
        torch.cuda.synchronize()
        ctx.pipeline(holos, indice=re, absorption=im)  # still queued when the capture begins
        batch = Batch([(ctx, holos, re, im, None)])
        ctx.synchronize()
        for _ in range(2):
            assert all(torch.equal(a, b) for a, b in zip(calls(ctx), want))
            re.zero_(), im.zero_()
            batch.launch()
            torch.cuda.synchronize()
            assert torch.equal(re, want[0]) and torch.equal(im, want[1])
        batch.close()
        assert all(torch.equal(a, b) for a, b in zip(calls(ctx), want))
