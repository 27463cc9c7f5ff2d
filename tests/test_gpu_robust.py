"""Device-side error reporting, in forms that fault nothing: a bounded wait made to run out by
lowering its poll budget, indices outside their segment, malformed packed offsets.  Each case
checks the status word, that the call returned, and that the next normal call is correct."""
import os

import numpy as np
import pytest
import torch

from oracle import oracle
from tests.util import assert_close_bf16, to_np

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lb():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lampa_b200
    return lampa_b200


def _status(lb):
    from lampa_b200 import _lib as L
    torch.cuda.synchronize()
    st = L.status_word(torch.device("cuda:0"))
    vals = st.tolist()
    st.zero_()
    return vals


@pytest.mark.parametrize("hier,T", [(True, 64 * 40), (False, 64 * 40), (True, 64 * 3)])
def test_wait_that_runs_out_sets_timeout_and_returns(lb, hier, T):
    from lampa_b200 import _lib as L, synth
    H, K, V = 2, 64, 64
    Lv = lb.num_levels_required(T)
    inp = synth.gdn_inputs(3, T, H, K, V, L=Lv, g_shift=-3.0)
    d = {k: v.to("cuda:0") for k, v in inp.items()}
    old = os.environ.pop("LAMPA_B200_CHECK", None)

    def run():
        if hier:
            return lb.chunk_h_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["lam"], d["beta"],
                                               use_qk_l2norm_in_kernel=True)[0]
        return lb.chunk_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["beta"], use_qk_l2norm_in_kernel=True)[0]

    try:
        _status(lb)
        assert L.lib().lampa_debug_set_poll_budget(0) == 0
        run()
        vals = _status(lb)                     # synchronises: the kernels came back
        assert vals[0] == L.ERR_TIMEOUT, vals
    finally:
        L.lib().lampa_debug_set_poll_budget(1 << 22)
        if old is not None:
            os.environ["LAMPA_B200_CHECK"] = old
    o = run()
    assert _status(lb)[0] == 0
    a = [inp[k][0].float().numpy() for k in ("q", "k", "v", "g", "beta")]
    ref = oracle.hgdn(*a, inp["lam"][0].numpy(), use_l2norm=True)[0] if hier else oracle.gdn_plain(*a, use_l2norm=True)[0]
    assert_close_bf16(to_np(o[0]), ref, "call after a timed-out one")


def test_indices_outside_their_segment_are_skipped_and_reported(lb):
    from lampa_b200 import _lib as L
    _status(lb)
    src = torch.arange(40, dtype=torch.float32, device="cuda:0").view(10, 4)
    perm = torch.tensor([1, 0, 3, 2, 4, 0, 1, 2, 3, 99], dtype=torch.int64, device="cuda:0")   # two segments of 5
    dst = lb.permute_rows(src, perm, nseg=2)
    vals = _status(lb)
    assert vals[0] == L.ERR_BOUNDS and vals[1] == 10 and vals[2] == 9
    assert torch.equal(dst[:9], src[[1, 0, 3, 2, 4, 5, 6, 7, 8]])
    bad = torch.tensor([[0, 1, -1, 3]], dtype=torch.int64, device="cuda:0")
    lb.invert_permutation(bad)
    assert _status(lb)[0] == L.ERR_BOUNDS
    keys = torch.arange(16, dtype=torch.int32, device="cuda:0")
    lb.segmented_sort(keys, seg_offsets=torch.tensor([0, 8, 40]))                    # second segment leaves the array
    assert _status(lb)[0] == L.ERR_BOUNDS
    good = lb.segmented_sort(keys.flip(0), seg_offsets=torch.tensor([0, 8, 16]))
    assert _status(lb)[0] == 0
    assert good.tolist() == list(range(7, -1, -1)) * 2


def test_malformed_packed_offsets(lb):
    from lampa_b200 import _lib as L, synth
    T, H, K, V = 640, 1, 64, 64
    inp = synth.gdn_inputs(4, T, H, K, V, L=12, g_shift=-3.0)
    d = {k: v.to("cuda:0") for k, v in inp.items()}
    # host-resident offsets are checked on the host
    with pytest.raises(ValueError):
        lb.chunk_h_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["lam"], d["beta"],
                                    cu_seqlens=torch.tensor([0, 700]), use_qk_l2norm_in_kernel=True)
    with pytest.raises(ValueError):
        lb.chunk_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["beta"], cu_seqlens=torch.tensor([-64, 0, 640]))
    with pytest.raises(ValueError):   # 640 tokens in one sequence need 7 + 4 levels
        lb.chunk_h_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["lam"][..., :9], d["beta"],
                                    cu_seqlens=torch.tensor([0, 640]), use_qk_l2norm_in_kernel=True)
    # device-resident offsets: the kernels empty the bad sequence and report it
    old = os.environ.pop("LAMPA_B200_CHECK", None)
    try:
        _status(lb)
        lb.chunk_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["beta"],
                                  cu_seqlens=torch.tensor([-64, 0, 640], device="cuda:0"))
        assert _status(lb)[0] == L.ERR_BOUNDS
        lb.chunk_h_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["lam"][..., :9].contiguous(), d["beta"],
                                    cu_seqlens=torch.tensor([0, 640], device="cuda:0"), use_qk_l2norm_in_kernel=True)
        assert _status(lb)[0] == L.ERR_LEVELS
    finally:
        if old is not None:
            os.environ["LAMPA_B200_CHECK"] = old


def test_forward_only_ops_refuse_autograd(lb):
    q = torch.zeros(1, 128, 2, 64, dtype=torch.bfloat16, device="cuda:0", requires_grad=True)
    g = torch.zeros(1, 128, 2, device="cuda:0")
    with pytest.raises(NotImplementedError):
        lb.chunk_gated_delta_rule(q, q, q, g, g)
    with torch.no_grad():
        o, _ = lb.chunk_gated_delta_rule(q, q, q, g, g)
    assert not o.requires_grad


def test_sort_of_overlapping_segments_stays_inside_them(lb):
    """Offsets that fall make two segments of several tiles overlap: their passes rewrite each other's keys, the falling
    one between them is reported, and nothing is written behind the permutation or the workspace."""
    import ctypes
    from lampa_b200 import _lib as L
    n, pad = 400_000, 300_000
    rng = np.random.default_rng(9)
    keys = torch.from_numpy(rng.integers(-2**31, 2**31 - 1, n).astype(np.int32)).cuda()
    seg = torch.tensor([0, 300_000, 100_000, n], dtype=torch.int64, device="cuda:0")
    need = ctypes.c_size_t(0)
    L.check(L.lib().lampa_segsort_workspace_bytes(n, ctypes.byref(need)), "workspace")
    perm = torch.full((n + pad,), -7, dtype=torch.int64, device="cuda:0")
    ws = torch.full((need.value + 4 * pad,), 0x5A, dtype=torch.uint8, device="cuda:0")
    _status(lb)
    st = L.status_word(torch.device("cuda:0"))
    for _ in range(20):
        L.check(L.lib().lampa_segsort_stable(L.ptr(keys), L.LAMPA_KEY_I32, n, L.ptr(seg), 3, None, L.ptr(perm), L.ptr(ws), need.value,
                                             L.ptr(st), L.stream_ptr(torch.device("cuda:0"))), "lampa_segsort_stable")
    vals = _status(lb)
    assert vals[0] == L.ERR_BOUNDS and vals[1] == 12 and vals[2] == 1
    assert bool((perm[n:] == -7).all()) and bool((ws[need.value:] == 0x5A).all())


@pytest.mark.parametrize("bucket,dq,dv", [(100, 30, 24), (25, 30, 24), (50, 41, 40)])
def test_bucket_positions_outside_the_hits(lb, bucket, dq, dv):
    """Bucket positions that leave the hits are reported and not followed, on the tensor-core kernel and the FMA one (small
    buckets, wide rows with whole and ragged pieces): the other buckets' rows come out as without them."""
    from lampa_b200 import _lib as L
    heads, n = 2, 4 * bucket
    gen = torch.Generator().manual_seed(bucket)
    q, k = (torch.randn(heads, n, dq, generator=gen).cuda() * 0.3 for _ in range(2))
    v = torch.randn(heads, n, dv, generator=gen).cuda()
    qp, kp = (torch.stack([torch.randperm(n, generator=gen) for _ in range(heads)]).unsqueeze(0).cuda() for _ in range(2))
    want = lb.hept_bucket_attention(q, k, v, qp, kp, bucket)
    old = os.environ.pop("LAMPA_B200_CHECK", None)
    try:
        assert _status(lb)[0] == 0
        for which in (qp, kp):
            bad = which.clone()
            bad[0, 0, :3] = torch.tensor([n, -1, 1 << 40])              # first bucket of the first head
            got = lb.hept_bucket_attention(q, k, v, *((bad, kp) if which is qp else (qp, bad)), bucket)
            vals = _status(lb)
            assert vals[0] == L.ERR_BOUNDS and vals[1] == 50 and vals[2] < 3
            assert torch.equal(got[1], want[1])
            others = qp[0, 0, bucket:]
            others = others[others != 0]                               # a bad entry stands for hit 0
            assert torch.equal(got[0][others], want[0][others])
    finally:
        if old is not None:
            os.environ["LAMPA_B200_CHECK"] = old


@pytest.mark.parametrize("n,flat", [(300, False), (60_000, False), (300, True)])
def test_sort_starting_order_outside_its_segment(lb, n, flat):
    """Entries of a starting order that leave their segment are reported and stand for its first element (`flat`: all keys are
    equal and no pass is needed); the other segment is sorted as ever."""
    from lampa_b200 import _lib as L
    rng = np.random.default_rng(31)
    keys = np.zeros(2 * n, np.float32) if flat else rng.standard_normal(2 * n).astype(np.float32)
    init = np.stack([rng.permutation(n) for _ in range(2)])
    bad = init.copy()
    bad[1, [3, 17, n - 1]] = [n, -1, 1 << 40]
    _status(lb)
    got = to_np(lb.segmented_sort(torch.from_numpy(keys).cuda(), nseg=2, init=torch.from_numpy(bad.reshape(-1)).cuda()))
    vals = _status(lb)
    assert vals[0] == L.ERR_BOUNDS and vals[1] == 14 and vals[2] == 1
    bad[1, [3, 17, n - 1]] = 0
    for s in range(2):
        k = keys[s * n:(s + 1) * n][bad[s]]
        np.testing.assert_array_equal(got[s * n:(s + 1) * n], bad[s][np.argsort(k, kind="stable")])


@pytest.mark.parametrize("K,hier", [(64, False), (64, True), (32, True)])
def test_sequences_that_overlap_are_emptied(lb, K, hier):
    """Offsets that fall and rise again: a sequence that begins before an earlier offset is emptied and reported, since its
    chunks have no records, and the sequences in order give what they give alone."""
    from lampa_b200 import _lib as L, synth
    T, H = 640, 2
    inp = synth.gdn_inputs(6, T, H, K, K, L=11, g_shift=-3.0)
    d = {k: v.to("cuda:0") for k, v in inp.items()}
    old = os.environ.pop("LAMPA_B200_CHECK", None)

    def run(cu):
        c = torch.tensor(cu, device="cuda:0")
        if hier:
            return lb.chunk_h_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["lam"], d["beta"], cu_seqlens=c,
                                               use_qk_l2norm_in_kernel=True)[0], None
        return lb.chunk_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["beta"], cu_seqlens=c, output_final_state=True,
                                         use_qk_l2norm_in_kernel=True)

    try:
        _status(lb)
        want, state = run([0, T])
        assert _status(lb)[0] == 0
        for cu in ([0, T, 0, T], [0, T, 64, T, 128, T, 0, T]):
            got, st = run(cu)
            vals = _status(lb)
            assert vals[0] == L.ERR_BOUNDS and vals[1] == 1, vals
            assert torch.equal(got, want)
            assert st is None or (torch.equal(st[0], state[0]) and not st[1:].any())
        # behind an offset that leaves the input, sequences in order are taken as before
        got, _ = run([0, 256, T + 64, 320, T])
        want, _ = run([0, 256, 256, 320, T])
        assert torch.equal(got[:, :256], want[:, :256]) and torch.equal(got[:, 320:], want[:, 320:])
        assert _status(lb)[0] == L.ERR_BOUNDS
        # more sequences than the plan takes in one pass
        cu = list(range(0, 600, 2)) + [T]
        want, _ = run(cu)
        assert _status(lb)[0] == 0
        cu[290] = 10
        got, _ = run(cu)
        assert torch.equal(got[:, :578], want[:, :578]) and torch.equal(got[:, 582:], want[:, 582:])
        assert _status(lb)[0] == L.ERR_BOUNDS
    finally:
        if old is not None:
            os.environ["LAMPA_B200_CHECK"] = old


def _model(lb, n):
    from lampa_b200 import synth
    from lampa_b200.model import LSHGatedDelta
    torch.manual_seed(5)
    return LSHGatedDelta(max_hits_per_event=4096, n_layers=3).to("cuda:0"), synth.detector_hits(17, n).to("cuda:0")


@pytest.mark.parametrize("over", [50, 1 << 40])
def test_model_rows_of_events_outside_the_input_are_skipped(lb, over):
    """Device-resident event offsets whose inner entry lies behind or before the rows: no row is followed out of the
    input, no block adds anything to a skipped row, and the call reports it."""
    from lampa_b200 import _lib as L
    n = 700
    m, hits = _model(lb, n)
    old = os.environ.pop("LAMPA_B200_CHECK", None)
    try:
        _status(lb)
        with torch.no_grad():
            x = m.head(m.encoder(hits * m.feature_scale))
        for cu in ([0, n + over, n], [0, -over, n]):
            got = m(hits, torch.tensor(cu, device="cuda:0"))
            assert _status(lb)[0] == L.ERR_BOUNDS
            # fp32 sums of 24 and 128 terms in another order
            torch.testing.assert_close(got, x, rtol=1e-5, atol=1e-5)
        m(hits, torch.tensor([0, n], device="cuda:0"))
        assert _status(lb)[0] == 0
    finally:
        if old is not None:
            os.environ["LAMPA_B200_CHECK"] = old


@pytest.mark.parametrize("bad", [[0, 300, 1200, 700], [-250, 0, 300, 700], [0, 300, -1, 700]])
def test_model_events_beside_a_bad_one_are_unchanged(lb, bad):
    """The orders of all rounds are one segmented sort: an offset that leaves the batch reaches into no other segment, and the
    first event's 300 rows come out as they do beside a good one."""
    from lampa_b200 import _lib as L
    n = 700
    m, hits = _model(lb, n)
    old = os.environ.pop("LAMPA_B200_CHECK", None)
    try:
        _status(lb)
        good = torch.tensor([0, 300, n], device="cuda:0")
        want, order = m(hits, good), m.orderings(hits, good)
        assert _status(lb)[0] == 0
        cu = torch.tensor(bad, device="cuda:0")
        for _ in range(10):
            got, perm = m(hits, cu), m.orderings(hits, cu)
            assert torch.equal(perm[:, :300], order[:, :300]) and torch.equal(got[:300], want[:300])
        assert _status(lb)[0] == L.ERR_BOUNDS
    finally:
        if old is not None:
            os.environ["LAMPA_B200_CHECK"] = old


def test_short_conv_of_sequences_outside_the_input(lb):
    """Device-resident offsets in front of and behind the rows: taps and final-state slots outside the input are zero."""
    T, D, W = 100, 32, 4
    conv = lb.ShortConvolution(D, W, device="cuda:0", dtype=torch.float32)
    x = torch.randn(1, T, D, device="cuda:0")
    want, _ = conv(x, cu_seqlens=torch.tensor([0, 40, T], device="cuda:0"))
    got, state = conv(x, cu_seqlens=torch.tensor([-(1 << 36), 40, 1 << 40], device="cuda:0"), output_final_state=True)
    assert torch.equal(got, want)                               # all rows have the taps of the sequence they lie in
    assert torch.equal(state[0], x[0, 40 - W:40].T) and not state[1].any()


def _model_structs(m):
    """The two C structs of a model's first block, and what they point to."""
    import ctypes
    vp = ctypes.c_void_p

    class Mixer(ctypes.Structure):
        _fields_ = [(n, vp) for n in ("q_w", "k_w", "v_w", "g_w", "a_w", "b_w", "l_w", "q_conv", "k_conv", "v_conv",
                                      "A_log", "dt_bias", "Lw")] + [("H", ctypes.c_int32), ("L", ctypes.c_int32)]

    class Update(ctypes.Structure):
        _fields_ = [(n, vp) for n in ("o_norm_w", "o_w", "up_w", "up_b", "down_w", "down_b", "mlp_norm_w", "next_norm_w")] + [
            (n, ctypes.c_float) for n in ("o_eps", "eps", "next_eps")] + [("head_dim", ctypes.c_int32)]

    b, at = m.blocks[0], m.blocks[0].attn
    mix = Mixer(*(t.data_ptr() for t in (at.q_proj.weight, at.k_proj.weight, at.v_proj.weight, at.g_proj.weight, at.a_proj.weight,
                                         at.b_proj.weight, at.l_proj.weight, at.q_conv1d.weight, at.k_conv1d.weight,
                                         at.v_conv1d.weight, at.A_log, at.dt_bias, at.L)), at.num_heads, at.num_levels)
    upd = Update(*(t.data_ptr() for t in (at.o_norm.weight, at.o_proj.weight, b.mlp_up.weight, b.mlp_up.bias, b.mlp_down.weight,
                                          b.mlp_down.bias, b.mlp_norm_weight, m.blocks[1].attn_norm_weight)),
                 at.o_norm.eps, b.eps, b.eps, at.head_dim)
    return mix, upd


@pytest.mark.parametrize("budget", [0, 1])
def test_model_kernels_whose_waits_run_out_return(lb, budget):
    """Both block kernels with several tiles per CTA: a wait that runs out is reported, the kernel drains and comes back, and
    the next call is right."""
    import ctypes
    from lampa_b200 import _lib as L
    n = 148 * 2 * 128 * 2 + 77                                  # every CTA has more than two tiles
    m, _ = _model(lb, 1)
    mix, upd = _model_structs(m)
    gen = torch.Generator(device="cuda").manual_seed(2)
    new = lambda *s, dt=torch.bfloat16: torch.randn(*s, generator=gen, device="cuda", dtype=torch.float32).to(dt)
    hs, o, gate = new(n, 128), new(n, 128), new(n, 128)
    x0 = new(n, 128, dt=torch.float32)
    perm = torch.randperm(n, generator=gen, device="cuda")
    cu = torch.tensor([0, n], device="cuda:0")
    st, stream = L.status_word(torch.device("cuda:0")), L.stream_ptr(torch.device("cuda:0"))
    lib = L.lib()
    vp = ctypes.c_void_p

    def project():
        out = [torch.empty(n, 128, dtype=torch.bfloat16, device="cuda:0") for _ in range(4)]
        out += [torch.empty(n, mix.H, device="cuda:0") for _ in range(2)]
        out += [torch.empty(n, mix.H * mix.L, dtype=torch.bfloat16, device="cuda:0")]
        L.check(lib.lampa_model_project(ctypes.byref(mix), vp(hs.data_ptr()), vp(perm.data_ptr()), vp(cu.data_ptr()), 1,
                                        ctypes.c_int64(n), *(vp(t.data_ptr()) for t in out), vp(st.data_ptr()), vp(stream)), "project")
        return out

    def update():
        x, y = x0.clone(), torch.empty_like(hs)
        L.check(lib.lampa_model_update(ctypes.byref(upd), vp(o.data_ptr()), vp(gate.data_ptr()), vp(x.data_ptr()), vp(perm.data_ptr()),
                                       vp(cu.data_ptr()), 1, ctypes.c_int64(n), vp(y.data_ptr()), vp(st.data_ptr()), vp(stream)), "update")
        return [x, y]

    _status(lb)
    for call, waits in ((project, range(600, 620)), (update, range(620, 640))):
        want = call()
        assert _status(lb)[0] == 0
        try:
            assert lib.lampa_debug_set_poll_budget(budget) == 0
            call()
            vals = _status(lb)
        finally:
            lib.lampa_debug_set_poll_budget(1 << 22)
        # a single poll may wait long enough in hardware to succeed
        assert vals[0] == L.ERR_TIMEOUT and vals[1] in waits if budget == 0 else vals[0] in (0, L.ERR_TIMEOUT)
        assert all(torch.equal(a, b) for a, b in zip(call(), want))
        assert _status(lb)[0] == 0


@pytest.mark.parametrize("counted", [True, False])
@pytest.mark.parametrize("budget", [0, 1])
def test_decode_step_whose_wait_runs_out_leaves_the_counts(lb, counted, budget):
    """The one-launch step and the one with a launch of its own for the counts: slabs that did not arrive in time are not
    stepped, and then the counts are not either; the arrival counter is zero again for the next step."""
    import ctypes
    from lampa_b200 import _lib as L, synth
    B, H, K, Lv = 16, 4, 64, 13
    inp = {k: v.to("cuda:0") for k, v in synth.gdn_inputs(8, B, H, K, K, L=Lv, g_shift=-3.0).items()}
    x = {k: v[0].contiguous() for k, v in inp.items()}                     # B rows of one token
    gen = torch.Generator(device="cuda").manual_seed(1)
    states = torch.randn(B, H, K, K, Lv, generator=gen, device="cuda")
    counts = torch.tensor([1, 1, 2, 0, 8] + [0] * (Lv - 5), dtype=torch.int32, device="cuda:0")
    arrivals = torch.zeros(1, dtype=torch.int32, device="cuda:0")
    desc = L.GdnDesc(B=B, T=1, H=H, K=K, V=K, L=Lv, nseq=0, qkv_dtype=L.dtype_code(x["q"].dtype), gb_dtype=L.dtype_code(x["g"].dtype),
                     lam_dtype=L.dtype_code(x["lam"].dtype), use_l2norm=1, scale=1.0)
    st, stream = L.status_word(torch.device("cuda:0")), L.stream_ptr(torch.device("cuda:0"))

    def step(s, c):
        o = torch.empty_like(x["v"])
        a = [L.ptr(x[k]) for k in ("q", "k", "v", "g", "beta", "lam")] + [L.ptr(s), L.ptr(c)]
        if counted:
            rc = L.lib().lampa_hgdn_step_counted(ctypes.byref(desc), *a, L.ptr(arrivals), L.ptr(o), L.ptr(st), stream)
        else:
            rc = L.lib().lampa_hgdn_step(ctypes.byref(desc), *a, L.ptr(o), L.ptr(st), stream)
        L.check(rc, "step")
        return o

    _status(lb)
    want_s, want_c = states.clone(), counts.clone()
    want = step(want_s, want_c)
    assert _status(lb)[0] == 0 and want_c.tolist()[:5] == [1, 0, 0, 4, 8]
    s, c = states.clone(), counts.clone()
    try:
        assert L.lib().lampa_debug_set_poll_budget(budget) == 0
        step(s, c)
        vals = _status(lb)
    finally:
        L.lib().lampa_debug_set_poll_budget(1 << 22)
    assert arrivals.item() == 0
    if budget == 0:
        assert vals[0] == L.ERR_TIMEOUT and vals[1] == 32
        assert torch.equal(s, states)
    assert torch.equal(c, counts if vals[0] == L.ERR_TIMEOUT else want_c)    # one poll may wait long enough to succeed
    s, c = states.clone(), counts.clone()
    o = step(s, c)
    assert _status(lb)[0] == 0 and arrivals.item() == 0
    assert torch.equal(o, want) and torch.equal(s, want_s) and torch.equal(c, want_c)
