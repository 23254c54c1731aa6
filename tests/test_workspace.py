"""The engine's workspace when there is little of it: a limit set by the
caller, or a device that is nearly full."""
import ctypes

import numpy as np
import pytest

from libnegf_b200 import generators as G
from libnegf_b200 import native

pytestmark = pytest.mark.gpu


def _layout(n, nbl, npts):
    """Bytes of a point's slots, of the blocks kept between the launches of a
    split call, and of one launch of whole points (at most two CTAs an SM)."""
    per = (15 + 2 + nbl + 2) * 16 * n * n
    return per, 2 * npts * 16 * n * n


def test_a_tight_limit_keeps_the_teams_of_the_sweeps(gpu_ctx):
    """The contacts' blocks of a split call count against the limit: where they
    would leave fewer teams for the points than one launch of whole points
    has, the call is not split."""
    n, nbl, npts = 48, 2, 1000
    per, blocks = _layout(n, nbl, npts)
    h = gpu_ctx.upload(G.transport_c0(nbl=nbl, n=n, seed=3))
    E = np.linspace(-1.0, 1.0, npts)
    try:
        gpu_ctx.set_options(schedule=1)
        n0 = gpu_ctx.launch_count()
        T, nc, st = gpu_ctx.transmission(h, E, eta=1e-3)
        assert gpu_ctx.launch_count() - n0 >= 2
        gpu_ctx.set_workspace_limit(blocks + 8 * per)
        n0 = gpu_ctx.launch_count()
        Tl, nl, sl = gpu_ctx.transmission(h, E, eta=1e-3)
        assert gpu_ctx.launch_count() - n0 == 1
        assert np.array_equal(Tl, T) and np.array_equal(nl, nc) and np.array_equal(sl, st)
    finally:
        gpu_ctx.set_workspace_limit(0)
        gpu_ctx.set_options()
        gpu_ctx.release(h)


def test_a_call_runs_where_only_its_whole_points_fit():
    """Without a limit, on a device with room for the slots of whole points but
    not for the blocks of a split call besides: the call runs as one launch."""
    torch = pytest.importorskip("torch")
    n, nbl, npts = 128, 2, 1000
    per, blocks = _layout(n, nbl, npts)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    whole = 2 * sms * per
    dev = G.transport_c0(nbl=nbl, n=n, seed=3)
    E = np.linspace(-1.0, 1.0, npts)
    with native.Context(0) as ctx:
        h = ctx.upload(dev)
        T, nc, st = ctx.transmission(h, E[:20], eta=1e-3)
    torch.cuda.empty_cache()
    with native.Context(0) as ctx:
        h = ctx.upload(dev)
        free = torch.cuda.mem_get_info()[0]
        fill = torch.empty(free - whole - blocks // 2, dtype=torch.uint8, device="cuda")
        try:
            n0 = ctx.launch_count()
            Tl, nl, sl = ctx.transmission(h, E, eta=1e-3)
            assert ctx.launch_count() - n0 == 1
        finally:
            del fill
            torch.cuda.empty_cache()
    assert np.array_equal(Tl[:20], T) and np.array_equal(nl[:20], nc) and np.all(sl == 0)


def test_a_captured_call_takes_the_workspace_in_place():
    """The same device: after an eager call a captured one, whose split plan
    would need to grow the workspace, runs whole points in the one in place."""
    torch = pytest.importorskip("torch")
    n, nbl, npts = 128, 2, 1000
    per, blocks = _layout(n, nbl, npts)
    whole = 2 * torch.cuda.get_device_properties(0).multi_processor_count * per
    E = np.linspace(-1.0, 1.0, npts)
    L = native.load()
    torch.cuda.empty_cache()
    with native.Context(0) as ctx:
        h = ctx.upload(G.transport_c0(nbl=nbl, n=n, seed=3))
        d_ids = torch.full((npts,), h, dtype=torch.int32, device="cuda")
        d_E = torch.from_numpy(E).cuda()
        d_T = torch.zeros(npts, dtype=torch.float64, device="cuda")
        d_nc, d_st = torch.zeros((2, npts), dtype=torch.int32, device="cuda")
        s = torch.cuda.Stream()

        def call():
            return L.negf_b200_transmission_dev(ctx.handle, npts, d_ids.data_ptr(), d_E.data_ptr(), 1e-3, 1, 2,
                                                d_T.data_ptr(), d_nc.data_ptr(), d_st.data_ptr(),
                                                ctypes.c_void_p(s.cuda_stream))

        fill = torch.empty(torch.cuda.mem_get_info()[0] - whole - blocks // 2, dtype=torch.uint8, device="cuda")
        try:
            assert call() == 0
            s.synchronize()
            T, nc = d_T.cpu().numpy(), d_nc.cpu().numpy()
            d_T.zero_()
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                rc = call()
            assert rc == 0
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(d_T.cpu().numpy(), T) and np.array_equal(d_nc.cpu().numpy(), nc)
            assert not bool(d_st.any())
            del g
        finally:
            del fill
            torch.cuda.empty_cache()


def test_a_call_that_succeeds_leaves_no_message(gpu_ctx):
    """A small-order call needs no workspace of the engine; a limit that would
    refuse the engine is none of its errors."""
    with native.Context(0) as ctx:
        h = ctx.upload(G.transport_c0(nbl=4, n=8, seed=2))
        ctx.set_workspace_limit(15 * 16 * 8 * 8)
        T, nc, st = ctx.transmission(h, np.linspace(-1, 1, 5), eta=1e-3)
        assert np.all(st == 0) and ctx.last_error() == ""
