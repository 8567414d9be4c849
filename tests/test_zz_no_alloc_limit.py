"""The allocation-free entry point takes every view count up to its limit: small
frames of 55 views, of the counts after it and of the limit itself equal
stratum_renderViews bit for bit (the views share one table; each has its own
camera and frame buffers)."""
import ctypes as ct

import pytest
import torch

import stratum_hyperdetail_b200 as sb

pytestmark = pytest.mark.gpu
W, H = 24, 17


def many_views(view, n):
    """A device table of n views of one world, turned a little each, and their buffers."""
    buf = {k: torch.zeros(n, W * H * (1 if k == "Pixels" else 4), device="cuda",
                          dtype=torch.int32 if k == "Pixels" else torch.float32)
           for k in ("Hit", "Surface", "Linear", "History", "Pixels")}
    C = view.C.repeat(n, 1)
    C[:, 3] += torch.arange(n, device="cuda") * 0.1
    rec = (sb.ViewRecord * n)()
    for i, r in enumerate(rec):
        for k in ("Origin", "I", "World", "Tags", "Nodes", "Queue"):
            setattr(r, k, sb.ptr(getattr(view, k)))
        r.C = sb.ptr(C[i])
        for k, t in buf.items():
            setattr(r, k, sb.ptr(t[i]))
        r.width, r.height = W, H
    return torch.frombuffer(bytearray(bytes(rec)), dtype=torch.uint8).cuda(), buf, C


@pytest.mark.parametrize("n", [55, 56, sb.NOALLOC_MAX_VIEWS - 1, sb.NOALLOC_MAX_VIEWS])
def test_no_alloc_takes_every_count_up_to_its_limit(cuda, n):
    from stratum_hyperdetail_b200.views import View
    v = View(W, H)
    v.set_pose(5, (3, 0, 4, 0), (17.0, 30.0, 0.0), 0.6, -0.3)
    v.C[19] = 1.0
    s = torch.cuda.current_stream().cuda_stream
    table, want, keep = many_views(v, n)
    size = int(sb.lib().stratum_batchScratchBytes(n))
    scratch = torch.zeros(size, dtype=torch.uint8, device="cuda")
    tune = sb.Tune(128, 1, 1)
    sb.call("stratum_renderViews", sb.ptr(table), n, sb.ptr(scratch), size, ct.byref(tune), s)
    table2, got, keep2 = many_views(v, n)
    sb.call("stratum_renderViewsNoAlloc", sb.ptr(table2), n, ct.byref(tune), s)
    torch.cuda.synchronize()
    for k in want:
        assert torch.equal(got[k], want[k]), k
    assert (want["Hit"][:, 1::4] >= 0).any(dim=1).all()  # every view shows something
