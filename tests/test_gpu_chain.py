"""Calls behind one another on a stream, without a synchronisation in between: a kernel may be resident before the one in
front of it is complete, and must neither read what that one still writes nor overwrite what it still reads."""
import pytest
import torch
import torch.nn.functional as F

import lampa_b200

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def unchecked(monkeypatch):
    """No look at the status word behind each call, which other test modules ask for: it synchronises, and cannot be captured."""
    monkeypatch.setenv("LAMPA_B200_CHECK", "0")


def _inputs(seed, B, T, H, K, V, L):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    return [rn(B, T, H, K).bfloat16(), rn(B, T, H, K).bfloat16(), rn(B, T, H, V).bfloat16(), -F.softplus(rn(B, T, H) - 3),
            torch.sigmoid(rn(B, T, H)), F.softplus(rn(B, T, H, L)).bfloat16()]


def _mixer(x, **kw):
    q, k, v, g, beta, lam = x
    return lampa_b200.chunk_h_gated_delta_rule(q, k, v, g, lam, beta, use_qk_l2norm_in_kernel=True, **kw)


# (64 * 6 + 50 and 64 * 31 + 50 at head dims up to 32: a tail taken in at once behind two and five chunk levels)
@pytest.mark.parametrize("T,H,K,V", [(1, 2, 64, 64), (130, 3, 16, 32), (700, 4, 64, 64), (5003, 2, 32, 32), (64 * 6 + 50, 3, 32, 32), (64 * 31 + 50, 3, 16, 32)])
def test_inputs_rewritten_between_calls(T, H, K, V):
    """Each call's inputs are the same buffers, rewritten by torch and by the library's own gather right before it."""
    L = lampa_b200.num_levels_required(max(T, 64))
    sets = [_inputs(s, 1, T, H, K, V, L) for s in range(4)]
    order = torch.randperm(T, device="cuda", generator=torch.Generator(device="cuda").manual_seed(9))
    want = []
    for x in sets:
        y = [t.clone() for t in x]
        torch.cuda.synchronize()
        y[2] = lampa_b200.permute_rows(y[2].view(T, -1), order).view(1, T, H, V)
        torch.cuda.synchronize()
        o, st = _mixer(y, output_final_state=True)
        p, ht = lampa_b200.chunk_gated_delta_rule(*y[:5], output_final_state=True, use_qk_l2norm_in_kernel=True)
        torch.cuda.synchronize()
        want.append([t.clone() for t in (o, st.states, p, ht)])
    buf = [torch.empty_like(t) for t in sets[0]]
    got = []
    torch.cuda.synchronize()
    for _ in range(5):
        got.clear()
        for x in sets:
            for b, t in zip(buf, x):
                b.copy_(t)
            rows = lampa_b200.permute_rows(buf[2].view(T, -1), order).view(1, T, H, V)
            y = buf[:2] + [rows] + buf[3:]
            o, st = _mixer(y, output_final_state=True)
            p, ht = lampa_b200.chunk_gated_delta_rule(*y[:5], output_final_state=True, use_qk_l2norm_in_kernel=True)
            got.append((o, st.states, p, ht))
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            assert torch.equal(a, b)


def test_steps_behind_one_another():
    """Fifty decode steps on one state, each reading what the one before wrote."""
    H, K, V, L = 4, 32, 32, 17
    x0 = _inputs(1, 2, 128, H, K, V, L)
    steps = [_inputs(100 + i, 2, 1, H, K, V, L) for i in range(50)]
    runs = []
    for sync in (True, False):
        _, st = _mixer(x0, output_final_state=True)
        outs = []
        for x in steps:
            if sync:
                torch.cuda.synchronize()
            o, st = _mixer(x, initial_state=st, output_final_state=True)
            outs.append(o)
        runs.append((torch.stack(outs), st.states.clone(), st.counts.clone()))
    for a, b in zip(*runs):
        assert torch.equal(a, b)


def _prompts(T, H, K, V, n):
    L = lampa_b200.num_levels_required(max(T, 64))
    sets = [_inputs(20 + s, 1, T, H, K, V, L) for s in range(n)]
    want = []
    for x in sets:
        torch.cuda.synchronize()
        o, st = _mixer(x, output_final_state=True)
        torch.cuda.synchronize()
        want.append((o.clone(), st.states.clone(), st.counts.clone()))
    return sets, want


# a prompt whose tail is taken in at once, token by token, and none; more CTAs than fit the GPU
@pytest.mark.parametrize("T,H,K,V", [(700, 4, 64, 64), (3001, 8, 64, 64), (643, 4, 64, 64), (1024, 8, 64, 64), (5003, 2, 32, 32), (700, 40, 16, 32)])
def test_prefill_replayed(T, H, K, V):
    """The end of a prompt begins beside its output pass, in a replayed graph too, where every replay has the same number."""
    sets, want = _prompts(T, H, K, V, 3)
    buf = [t.clone() for t in sets[0]]
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        _mixer(buf, output_final_state=True)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            rows = [t + 0 for t in buf]                      # written right in front of the call
            o, st = _mixer(rows, output_final_state=True)
        got = []
        for _ in range(4):
            for x in sets:
                for b, t in zip(buf, x):
                    b.copy_(t)
                graph.replay()
                got.append((o.clone(), st.states.clone(), st.counts.clone()))
    torch.cuda.synchronize()
    for i, g in enumerate(got):
        for a, b in zip(g, want[i % 3]):
            assert torch.equal(a, b), i


@pytest.mark.parametrize("T,H,K,V", [(700, 4, 64, 64), (3001, 8, 64, 64), (5003, 2, 32, 32)])
def test_prefills_beside_one_another(T, H, K, V):
    """Prompts on three streams, their kernels among one another's on the same SMs; each writes its inputs right before its call."""
    sets, want = _prompts(T, H, K, V, 3)
    streams = [torch.cuda.Stream() for _ in sets]
    got = [[] for _ in sets]
    torch.cuda.synchronize()
    for _ in range(6):
        for i, (s, x) in enumerate(zip(streams, sets)):
            with torch.cuda.stream(s):
                o, st = _mixer([t + 0 for t in x], output_final_state=True)
                got[i].append((o, st.states, st.counts))
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        for r in g:
            for a, b in zip(r, w):
                assert torch.equal(a, b)
