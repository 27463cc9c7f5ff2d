"""Calls of other sizes from other threads: the shared memory that a kernel may have is set per kernel, not per launch."""
import ctypes
import threading

import pytest
import torch

import lampa_b200
from lampa_b200 import _lib as L, synth

pytestmark = pytest.mark.gpu


def _mixer(K, V, Lv):
    """A hierarchical forward pass of 640 tokens, as the C interface takes it."""
    T, H = 640, 2
    x = {k: v.cuda() for k, v in synth.gdn_inputs(5, T, H, K, V, L=Lv, g_shift=-3.0).items()}
    desc = L.GdnDesc(B=1, T=T, H=H, K=K, V=V, L=Lv, nseq=0, qkv_dtype=L.dtype_code(x["q"].dtype), gb_dtype=L.dtype_code(x["g"].dtype),
                     lam_dtype=L.dtype_code(x["lam"].dtype), use_l2norm=1, scale=1.0)
    size = ctypes.c_size_t(0)
    L.check(L.lib().lampa_gdn_workspace_bytes(ctypes.byref(desc), ctypes.byref(size)), "workspace")
    buf = torch.empty(size.value + 1024, dtype=torch.uint8, device="cuda")
    ws = buf[-buf.data_ptr() % 1024 :][: size.value]
    o = torch.empty_like(x["v"])
    keep = [buf, o, x]
    args = [ctypes.byref(desc)] + [L.ptr(x[k]) for k in ("q", "k", "v", "g", "beta", "lam")]
    return keep, o, lambda st, stream: L.lib().lampa_hgdn_fwd(*args, None, L.ptr(o), L.ptr(ws), ws.numel(), L.ptr(st), stream)


def _step(K, V, Lv):
    """A decode step of four rows."""
    B, H = 4, 2
    x = {k: v[0].cuda().contiguous() for k, v in synth.gdn_inputs(5, B, H, K, V, L=Lv, g_shift=-3.0).items()}
    desc = L.GdnDesc(B=B, T=1, H=H, K=K, V=V, L=Lv, nseq=0, qkv_dtype=L.dtype_code(x["q"].dtype), gb_dtype=L.dtype_code(x["g"].dtype),
                     lam_dtype=L.dtype_code(x["lam"].dtype), use_l2norm=1, scale=1.0)
    states, counts, o = torch.zeros(B, H, K, V, Lv, device="cuda"), torch.zeros(Lv, dtype=torch.int32, device="cuda"), torch.empty_like(x["v"])
    keep = [x, states, counts, o]
    args = [ctypes.byref(desc)] + [L.ptr(x[k]) for k in ("q", "k", "v", "g", "beta", "lam")] + [L.ptr(states), L.ptr(counts), L.ptr(o)]
    return keep, o, lambda st, stream: L.lib().lampa_hgdn_step(*args, L.ptr(st), stream)


@pytest.mark.parametrize("make,K,V,levels,calls", [(_mixer, 64, 64, (11, 40), 1500), (_mixer, 32, 32, (11, 40), 1500), (_step, 64, 64, (20, 40), 500)])
def test_two_threads_with_other_level_counts(make, K, V, levels, calls):
    dev = torch.device("cuda:0")
    st = L.status_word(dev)
    jobs = [(make(K, V, Lv), torch.cuda.Stream()) for Lv in levels]
    want = []
    for (keep, o, call), _ in jobs:
        if make is _mixer:                               # (a step goes on from its state)
            L.check(call(st, L.stream_ptr(dev)), "call")
            want.append(o.clone())
    torch.cuda.synchronize()
    codes = [set() for _ in jobs]

    def work(i):
        (keep, o, call), stream = jobs[i]
        for n in range(calls):
            codes[i].add(call(st, stream.cuda_stream))
            if n % 100 == 99:
                stream.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [{0}, {0}]
    for (keep, o, call), w in zip((j for j, _ in jobs), want):
        assert torch.equal(o, w)
    lampa_b200.check_status(dev)
