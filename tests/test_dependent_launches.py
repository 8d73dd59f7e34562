"""Kernels whose set-up overlaps the kernel before them (programmatic dependent launches): chains
enqueued without a pause, in which each kernel reads what the one before it wrote, give what the
same calls give one at a time."""
import numpy as np
import pytest
import torch

from mordred_b200 import _lib as L
from mordred_b200 import ssb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [999, 300_001])
def test_tables_rebuilt_between_queries(n):
    s = ssb.Sizes(lo_len=n, s_len=2_000, c_len=30_000, p_len=20_000)
    t = ssb.gen_device(s, 3, sorted(set(ssb.QA_FACT + ssb.QB_FACT)), sorted(set(ssb.QA_DIMS + ssb.QB_DIMS)))
    ws = ssb.StarWorkspace(s)
    asked = [(ssb.query_b, dict(c_region=i % 5, s_region=i % 3, mfgr=(i % 4, 4))) if i % 3 else
             (ssb.query_a, dict(category=i % 25, region=i % 5)) for i in range(60)]
    alone = []
    for query, kw in asked:
        alone.append(query(t, ws, **kw).clone())
        torch.cuda.synchronize()
    key = {k: t[k].long() for k in ("lo_suppkey", "lo_custkey", "lo_partkey", "lo_orderdate")}
    assert all(torch.equal(t[c], torch.arange(1, len(t[c]) + 1, device="cuda", dtype=torch.int32))
               for c in ("s_suppkey", "c_custkey", "p_partkey"))
    for (query, kw), got in zip(asked, alone):
        if query is ssb.query_b:
            m = (t["s_region"][key["lo_suppkey"] - 1] == kw["s_region"]) & \
                (t["c_region"][key["lo_custkey"] - 1] == kw["c_region"]) & \
                ((t["p_mfgr"][key["lo_partkey"] - 1] == kw["mfgr"][0]) | (t["p_mfgr"][key["lo_partkey"] - 1] == kw["mfgr"][1]))
            exp = (t["lo_revenue"][m].long() - t["lo_supplycost"][m].long()).sum()
        else:
            m = (t["s_region"][key["lo_suppkey"] - 1] == kw["region"]) & \
                (t["p_category"][key["lo_partkey"] - 1] == kw["category"])
            exp = t["lo_revenue"][m].long().sum()
        assert int(got.view(-1, 4)[:, 2:].contiguous().view(torch.int64).sum()) == int(exp)
    chained = [query(t, ws, **kw).clone() for query, kw in asked]
    torch.cuda.synchronize()
    for a, b in zip(alone, chained):
        assert torch.equal(a, b)


def test_training_steps_in_a_row():
    """Eight samples are one CTA's tile, so a step's sums have one order."""
    from mordred_b200.planner import init_params
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn(8, L.MB_MLP_IN, device="cuda", generator=g)
    target = torch.randn(8, L.MB_MLP_OUT, device="cuda", generator=g)
    ends = []
    for pause in (True, False):
        params = torch.from_numpy(init_params(2)).cuda()
        m, v, y = torch.zeros_like(params), torch.zeros_like(params), torch.zeros(8, L.MB_MLP_OUT, device="cuda")
        for step in range(1, 41):
            grads = torch.zeros_like(params)
            L.call("mb_mlp_backward", params.data_ptr(), x.data_ptr(), target.data_ptr(), 8, grads.data_ptr(), None,
                   ssb._stream())
            if pause:
                torch.cuda.synchronize()
            L.call("mb_mlp_adam", params.data_ptr(), grads.data_ptr(), m.data_ptr(), v.data_ptr(), params.numel(), 2e-3,
                   0.9, 0.999, 1e-8, step, 0.0, ssb._stream())
            if pause:
                torch.cuda.synchronize()
        L.call("mb_mlp_forward", params.data_ptr(), x.data_ptr(), 8, y.data_ptr(), ssb._stream())
        torch.cuda.synchronize()
        ends.append((params, y))
    assert torch.equal(ends[0][0], ends[1][0]) and torch.equal(ends[0][1], ends[1][1])
    assert np.isfinite(ends[0][1].cpu().numpy()).all()


def test_a_launch_that_fails_leaves_nothing_behind():
    """A launch on the legacy stream while another stream captures is refused by the runtime. The
    call says so; the next one, of a kernel that looks the last error up, is not refused for it."""
    import ctypes as C
    p = torch.zeros(64, device="cuda")
    key = torch.arange(1, 9, dtype=torch.int32, device="cuda")
    words = torch.zeros(16, dtype=torch.int32, device="cuda")
    adam = (p.data_ptr(), p.data_ptr(), p.data_ptr(), p.data_ptr(), 64, 1e-3, 0.9, 0.999, 1e-8, 1, 0.0, None)
    torch.cuda.synchronize()
    runtime = C.CDLL("libcudart.so.12")
    stream, graph = C.c_void_p(), C.c_void_p()
    assert runtime.cudaStreamCreate(C.byref(stream)) == 0
    assert runtime.cudaStreamBeginCapture(stream, 0) == 0  # global mode
    refused = L.lib().mb_mlp_adam(*adam)
    runtime.cudaStreamEndCapture(stream, C.byref(graph))
    runtime.cudaStreamDestroy(stream)
    runtime.cudaGetLastError()
    assert refused != L.MB_OK
    L.call("mb_pat_build", key.data_ptr(), 8, 0, 16, None, 0, None, 0, None, 0, words.data_ptr(), None)
    torch.cuda.synchronize()
    assert int((words != 0).sum()) == 8
