"""Volumes for host memory: index and absorption, one of them, or one beside a device buffer, equal those written to
device buffers bit for bit, also when queued calls rewrite the staged volumes before the earlier ones are read."""
import numpy as np
import pytest
import torch

from tests.helpers import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxmax,D", [(32, 128), (64, 256), (125, 512)])
def test_host_and_device_volumes(nxmax, D):
    from mtd_transmission_gb300 import Context, Geometry
    M = 6
    acq, _, d = small_case("plain_512_born", M=M, nxmax=nxmax, dim_final=D)

    def vol(where):
        if where is None:
            return None
        return torch.full((D, D, D), 7.0).pin_memory() if where == "host" else torch.full((D, D, D), 7.0, device="cuda")

    with Context(Geometry.from_acquisition(acq), M) as ctx:
        ctx.set_mask(np.ascontiguousarray(d["mask"]))
        stacks = [torch.from_numpy(np.ascontiguousarray(d["holos"][:n])).cuda() for n in (M, M - 2)]
        want = []
        for h in stacks:
            re, im = vol("device"), vol("device")
            torch.cuda.synchronize()
            ctx.pipeline(h, indice=re, absorption=im)
            ctx.synchronize()
            want.append((re.cpu(), im.cpu()))
        assert not torch.equal(want[0][0], want[1][0])
        forms = [("host", "host"), ("host", None), (None, "host"), ("host", "device"), ("device", "host"),
                 ("host", "host")]
        outs = [(vol(a), vol(b)) for a, b in forms]
        torch.cuda.synchronize()
        for k, (re, im) in enumerate(outs):
            ctx.pipeline_async(stacks[k % 2], indice=re, absorption=im)
        ctx.synchronize()
        for k, pair in enumerate(outs):
            for got, ref in zip(pair, want[k % 2]):
                assert got is None or torch.equal(got.cpu(), ref), forms[k]
