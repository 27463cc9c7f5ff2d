"""The end of a prompt (the last whole chunk's tokens and the T mod 64 behind it) is fp32 arithmetic up to the output's type:
prompts short enough that no chunk level has gone through a bf16 record, against the token recurrence in float64."""
import pytest
import torch
import torch.nn.functional as F

import lampa_b200

pytestmark = pytest.mark.gpu


def _fenwick64(q, k, v, g, b, lam):
    T, K = k.shape
    L = lam.shape[1]
    S = torch.zeros(L, K, v.shape[1], dtype=torch.float64)
    o = torch.zeros(T, v.shape[1], dtype=torch.float64)
    for t in range(T):
        if t:
            tz = (t & -t).bit_length() - 1
            S[tz + 1] += S[: tz + 1].sum(0)
            S[: tz + 1] = 0
        S = torch.exp(g[t]) * (S - b[t] * k[t][None, :, None] * (k[t] @ S)[:, None, :])
        S[0] += b[t] * torch.outer(k[t], v[t])
        o[t] = torch.einsum("l,k,lkv->v", lam[t], q[t], S)
    return o, S.permute(1, 2, 0)


# first and last token of a chunk, a chunk with nothing, one token and all but one behind it, fewer levels than a chunk has,
# more levels than the loads of one pass take (16), decays that leave nothing of a chunk; fp16 rows; tails on either side of 16 and
# 48, from where on they are taken in at once (64 and smaller head dims)
@pytest.mark.parametrize("K,V", [(64, 64), (32, 32), (16, 32)])
@pytest.mark.parametrize("T,L,shift,dt", [(1, 1, -3.0, torch.bfloat16), (4, 3, -3.0, torch.bfloat16), (63, 7, -3.0, torch.float16),
                                          (64, 9, -3.0, torch.bfloat16), (65, 9, 2.0, torch.bfloat16), (79, 9, -3.0, torch.bfloat16), (80, 9, -3.0, torch.float16),
                                          (127, 8, -3.0, torch.bfloat16),
                                          (100, 40, -5.0, torch.float16), (111, 9, -3.0, torch.bfloat16), (112, 17, -3.0, torch.bfloat16),
                                          (121, 40, -5.0, torch.float16), (126, 17, 2.0, torch.bfloat16)])
def test_short_prompts_are_fp32(K, V, T, L, shift, dt):
    B, H = 2, 3
    gen = torch.Generator().manual_seed(T * 64 + K)
    rn = lambda *s: torch.randn(*s, generator=gen)
    q, k, v = F.normalize(rn(B, T, H, K), dim=-1).to(dt), F.normalize(rn(B, T, H, K), dim=-1).to(dt), rn(B, T, H, V).to(dt)
    g, b, lam = -F.softplus(rn(B, T, H) + shift), torch.sigmoid(rn(B, T, H)), F.softplus(rn(B, T, H, L))
    o, st = lampa_b200.chunk_h_gated_delta_rule(q.cuda(), k.cuda(), v.cuda(), g.cuda(), lam.cuda(), b.cuda(),
                                                output_final_state=True, use_qk_l2norm_in_kernel=True)
    lampa_b200.check_status(torch.device("cuda:0"))
    kn = (k.float() * torch.rsqrt((k.float() ** 2).sum(-1, keepdim=True) + 1e-6)).to(dt)      # k is rounded, q is not
    qn = q.double() * torch.rsqrt((q.double() ** 2).sum(-1, keepdim=True) + 1e-6)
    n0 = T - T % 64
    for i in range(B):
        for h in range(H):
            ro, rs = _fenwick64(*(x[i, :, h].double() for x in (qn, kn, v, g, b, lam)))
            d = st.states[i, h].cpu().double() - rs
            # One decay factor is exp to two ulp, 2^-22.  At once (a tail of 16 or 48 tokens and more) an element goes through one such
            # factor and a few dozen roundings of 2^-24: four times 2^-22.  Token by token it goes through one factor per token, and
            # their errors may all point the same way.  (A whole chunk goes token by token too, at the tighter bound: it is within 0.65 of it.)
            bound = 2.0 ** -22 * (4 if T == n0 or T - n0 >= (16 if K == 64 else 48) else max(4, T))
            assert d.norm() <= bound * rs.norm(), (float(d.norm()), float(rs.norm()))
            if T > n0:
                e = o[i, n0:, h].cpu().double() - ro[n0:]
                eps = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11                          # rounding of the output, half an ulp
                assert (e.abs() <= eps * ro[n0:].abs() + 2 * bound * ro[n0:].abs().max()).all()
    want = [1 if T > 0 else 0] + [(1 << (l - 1)) if ((T - 1) >> (l - 1)) & 1 else 0 for l in range(1, L)]
    assert st.counts.view(-1)[:L].tolist() == want


# one chunk level live, two, an even number of chunks, five (one more than a batch of slots) and nine
@pytest.mark.parametrize("K,V", [(64, 64), (32, 32), (16, 32)])
@pytest.mark.parametrize("chunks,tail", [(2, 50), (5, 63), (6, 50), (31, 50), (511, 57)])
def test_a_tail_is_decode_steps(K, V, chunks, tail):
    """A tail taken in at once continues from the chunk levels as decode steps from the whole chunks' state do."""
    B, H, n0 = 2, 2, 64 * chunks
    T = n0 + tail
    L = lampa_b200.num_levels_required(T) + 1
    gen = torch.Generator(device="cuda").manual_seed(T + K)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x = [rn(B, T, H, K).bfloat16(), rn(B, T, H, K).bfloat16(), rn(B, T, H, V).bfloat16(), -F.softplus(rn(B, T, H) - 3), F.softplus(rn(B, T, H, L)),
         torch.sigmoid(rn(B, T, H))]

    def run(a, b, state=None):
        return lampa_b200.chunk_h_gated_delta_rule(*(t[:, a:b].contiguous() for t in x), initial_state=state, output_final_state=True,
                                                   use_qk_l2norm_in_kernel=True)

    o, st = run(0, T)
    _, steps = run(0, n0)
    start = steps.states.flatten(2).norm(dim=-1)              # per row and head
    outs = []
    for t in range(n0, T):
        ot, steps = run(t, t + 1, steps)
        outs.append(ot)
    lampa_b200.check_status(torch.device("cuda:0"))
    assert torch.equal(st.counts, steps.counts)
    # A token's transition is a contraction, entered with an error of a few 2^-24 and one decay factor to 2^-22: 2^-21 of the state
    # per token, of the steps and of the closed form, on states that grow by their token (at most |v|) each.
    bound = 2 * tail * 2.0 ** -21 * (start + x[2].float()[:, n0:].norm(dim=-1).amax(1))
    d = (st.states - steps.states).flatten(2, 3).norm(dim=2)        # per row, head and level
    assert (d <= bound[..., None]).all(), float((d / bound[..., None]).max())
    want = torch.cat(outs, 1).float()
    # both are rounded to bf16 (half a step each, 2^-8 of the value at most)
    lam = x[4][:, n0:].amax(-1)
    limit = 2.0 ** -7 * want.abs() + (x[0].float()[:, n0:].norm(dim=-1).clamp(max=1.0) * lam * L ** 0.5 * bound[:, None])[..., None]
    assert ((o[:, n0:].float() - want).abs() <= limit).all()


# a tail taken in at once behind a whole chunk, a prompt that is nothing but such a tail, and one that ends with a whole chunk; the
# token that carries the value: in the tail, its first one, one of the last whole chunk, the first of all
@pytest.mark.parametrize("K,V", [(64, 64), (32, 32), (16, 32)])
@pytest.mark.parametrize("T,n", [(121, 101), (121, 64), (121, 40), (57, 33), (57, 0), (64, 50), (700, 690)])
@pytest.mark.parametrize("what,value", [("q", "nan"), ("k", "nan"), ("k", "inf"), ("v", "nan"), ("v", "inf"), ("g", "nan"), ("g", "inf"), ("beta", "nan"),
                                        ("beta", "inf"), ("lam", "nan")])
def test_values_that_are_not_finite_reach_what_comes_after(K, V, T, n, what, value):
    """A NaN or an infinity at token n: outputs and states are finite exactly where the token recurrence has them finite, outputs in
    front of token n stay as they were, and so does the other head."""
    H, L = 2, 12
    gen = torch.Generator().manual_seed(T + K)
    rn = lambda *s: torch.randn(*s, generator=gen)
    x = dict(q=rn(1, T, H, K).bfloat16(), k=rn(1, T, H, K).bfloat16(), v=rn(1, T, H, V).bfloat16(), g=-F.softplus(rn(1, T, H) - 3),
             lam=F.softplus(rn(1, T, H, L)), beta=torch.sigmoid(rn(1, T, H)))

    def run():
        o, st = lampa_b200.chunk_h_gated_delta_rule(*(t.cuda() for t in x.values()), output_final_state=True, use_qk_l2norm_in_kernel=True)
        lampa_b200.check_status(torch.device("cuda:0"))
        return o[0].float().cpu(), st.states[0].cpu()

    o1, s1 = run()
    at = (0, n, 0, 3) if x[what].dim() == 4 else (0, n, 0)
    if what == "lam":
        at = (0, n, 0, 0)                                    # the level of the token itself, which every output reads
    x[what][at] = float(value)
    o2, s2 = run()
    # what the recurrence makes of it: the first and last of the tokens whose states are lost, and the outputs, which read all states
    lost = {"q": None, "lam": None, "v": (n, n), "k": (0, n), "beta": (0, n), "g": (0, n - 1) if n > 0 else None}[what]
    rows, cols = torch.zeros(T, V, dtype=torch.bool), slice(3, 4) if what == "v" else slice(None)
    rows[n : T if lost else n if what == "g" else n + 1, cols] = True
    # tokens of level l of the state: the older ones higher up, 2^(l-1) where bit l - 1 of T - 1 is set
    want, end = torch.zeros(K, V, L, dtype=torch.bool), 0
    for l in range(L - 1, -1, -1):
        size = 1 if l == 0 else (1 << (l - 1)) if ((T - 1) >> (l - 1)) & 1 else 0
        if size and lost and end <= lost[1] and lost[0] < end + size:
            want[:, cols, l] = True
        end += size
    n0 = T - T % 64                                          # outputs of whole chunks are not the tail's
    assert torch.equal(~torch.isfinite(o2[n0:, 0]), rows[n0:])
    assert torch.equal(~torch.isfinite(s2[0]), want)
    # what stays finite is what it was
    assert torch.equal(s2[1], s1[1]) and torch.equal(o2[n0:, 1], o1[n0:, 1])
    assert torch.equal(o2[n0:, 0][~rows[n0:]], o1[n0:, 0][~rows[n0:]])
    assert torch.equal(s2[0][~want], s1[0][~want])


# in the tail, taken in at once (64 x 64) and token by token, with no whole chunk, one, and several chunk levels in front
@pytest.mark.parametrize("K,V", [(64, 64), (32, 32)])
@pytest.mark.parametrize("T", [40, 57, 114, 64 * 7 + 40])
def test_a_decay_of_minus_infinity_forgets(T, K, V):
    """Whatever came before a token with g = -inf is gone, and nothing else changes.  (The tail's own arithmetic: whole chunks go
    through the chunkwise kernels, which take finite decays.)"""
    H, L = 2, 12
    gen = torch.Generator(device="cuda").manual_seed(T)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    n0, n = T - T % 64, T - 20
    x = [rn(1, T, H, K).bfloat16(), rn(1, T, H, K).bfloat16(), rn(1, T, H, V).bfloat16(), -F.softplus(rn(1, T, H)), F.softplus(rn(1, T, H, L)),
         torch.sigmoid(rn(1, T, H))]
    assert n >= n0
    run = lambda: lampa_b200.chunk_h_gated_delta_rule(*x, output_final_state=True, use_qk_l2norm_in_kernel=True)
    x[3][:, n] = -200.0                                      # e^-200 is zero in fp32
    o1, s1 = run()
    x[3][:, n] = float("-inf")
    o2, s2 = run()
    assert torch.isfinite(o2).all() and torch.isfinite(s2.states).all()
    assert torch.equal(o1, o2) or (o1.float() - o2.float()).norm() <= 1e-2 * o1.float().norm()
    assert (s1.states - s2.states).norm() <= 1e-6 * s1.states.norm()
    for i in (1, 2):                                         # other keys and values before token n
        x[i][:, :n] = rn(*x[i][:, :n].shape).bfloat16()
    o3, s3 = run()
    assert not torch.equal(o3[:, :n], o2[:, :n])
    # Forgotten to the bit where a decay enters as a factor.  The closed form multiplies the differences of running sums that are
    # -1e5 apart: e^-1e5 is zero too.
    assert torch.equal(o3[:, n:], o2[:, n:]) and torch.equal(s3.states, s2.states)


# one tiled copy per slab up to 32 levels, row by row beyond; more slabs than fit the GPU at once, and few
@pytest.mark.parametrize("K,V,H,B,L", [(64, 64, 4, 10, 17), (64, 64, 1, 37, 32), (64, 64, 1, 37, 33), (32, 32, 4, 19, 9), (16, 32, 8, 12, 17)])
def test_steps_of_large_batches(K, V, H, B, L):
    """Every row of a batch is stepped as it is alone, bit for bit."""
    gen = torch.Generator(device="cuda").manual_seed(B)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")

    def draw(T):
        return (rn(B, T, H, K).bfloat16(), rn(B, T, H, K).bfloat16(), rn(B, T, H, V).bfloat16(), -F.softplus(rn(B, T, H) - 3),
                F.softplus(rn(B, T, H, L)), torch.sigmoid(rn(B, T, H)))

    def run(x, state=None):
        return lampa_b200.chunk_h_gated_delta_rule(*x, initial_state=state, output_final_state=True, use_qk_l2norm_in_kernel=True)

    prompt, steps = draw(70), [draw(1) for _ in range(5)]
    _, state = run(prompt)
    rows = [run([t[i : i + 1].contiguous() for t in prompt])[1] for i in range(B)]
    for x in steps:
        o, state = run(x, state)
        for i in range(B):
            oi, rows[i] = run([t[i : i + 1].contiguous() for t in x], rows[i])
            assert torch.equal(o[i], oi[0]) and torch.equal(state.states[i], rows[i].states[0])
    lampa_b200.check_status(torch.device("cuda:0"))
