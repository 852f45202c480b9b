"""What tdm_autotune tries and leaves, seen through the number of launches: every schedule takes a known number of
launches a volume, and the autotuner runs each one it tries three times."""
import numpy as np
import pytest

from tests.helpers import small_case

pytestmark = pytest.mark.gpu

CAP, N = 112, 85  # scratch of 112 angles: chunks of 28 from host memory, 56 from device memory
LISTED = [(16, 4), (16, 2), (8, 4), (12, 4), (32, 2), (16, 6)]  # (32, 4) does not fit


def _launches(ctx, holos):
    before = ctx.launch_count
    ctx.pipeline(holos)
    ctx.synchronize()
    return ctx.launch_count - before


def _setup():
    import torch
    from mtd_transmission_gb300 import Context, Geometry
    acq, _, d = small_case("plain_512_born", M=N)
    host = torch.from_numpy(np.ascontiguousarray(d["holos"])).pin_memory()
    dev = host.cuda()
    torch.cuda.synchronize()
    return Geometry.from_acquisition(acq), Context, host, dev


def test_tries_the_present_schedule_and_leaves_the_host_one():
    geom, Context, host, dev = _setup()
    with Context(geom, CAP) as ctx, Context(geom, CAP) as other:
        usual, usual_host = _launches(ctx, dev), _launches(ctx, host)
        per = {}
        for s in LISTED + [(16, 1)]:
            other.set_schedule(*s)
            per[s] = _launches(other, dev)
        assert len({usual, usual_host, per[(16, 4)], per[(8, 4)], per[(12, 4)]}) == 5  # the counts tell them apart
        before = ctx.launch_count
        chunk = ctx.autotune(dev)
        assert ctx.launch_count - before == 3 * (usual + sum(per[s] for s in LISTED))
        assert chunk in {s[0] for s in LISTED}
        assert _launches(ctx, dev) in {usual} | {per[s] for s in LISTED}
        assert _launches(ctx, host) == usual_host
        # a schedule of the caller's own is tried too, beside the default
        ctx.set_schedule(16, 1)
        before = ctx.launch_count
        ctx.autotune(dev)
        assert ctx.launch_count - before == 3 * (usual + per[(16, 1)] + sum(per[s] for s in LISTED))


def test_error_leaves_the_schedules():
    from mtd_transmission_gb300.api import TdmError
    geom, Context, host, dev = _setup()
    with Context(geom, CAP) as ctx:
        counts = _launches(ctx, dev), _launches(ctx, host)
        ctx.set_wait_limit(0)  # every first wait of the extraction runs out: the call reports an error
        with pytest.raises(TdmError):
            ctx.autotune(dev)
        ctx.set_wait_limit(-1)
        assert (_launches(ctx, dev), _launches(ctx, host)) == counts
