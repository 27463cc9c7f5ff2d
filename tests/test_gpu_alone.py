"""A sequence's results depend on the sequence alone: the same bits by itself, in a batch, packed with others and in a slice of
its heads, on both sides of every rule that chooses a kernel by what a call carries as a whole (one CTA to an SM: 148 on a B200)."""
import pytest
import torch
import torch.nn.functional as F

import lampa_b200

pytestmark = pytest.mark.gpu


def _draw(seed, T, H, K, V, L):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    return [rn(1, T, H, K).bfloat16(), rn(1, T, H, K).bfloat16(), rn(1, T, H, V).bfloat16(), -F.softplus(rn(1, T, H) - 6),
            F.softplus(rn(1, T, H, L)).bfloat16(), torch.sigmoid(rn(1, T, H))]


def _hier(x, cu=None, state=False):
    return lampa_b200.chunk_h_gated_delta_rule(*x, cu_seqlens=cu, output_final_state=state, use_qk_l2norm_in_kernel=True)


def _plain(x, cu=None):
    return lampa_b200.chunk_gated_delta_rule(*x[:4], x[5], cu_seqlens=cu, output_final_state=True, use_qk_l2norm_in_kernel=True)


def _heads(x, a, b):
    return [t[:, :, a:b].contiguous() for t in x]


# two chunks; 141 chunks in blocks of eight (8 levels); 300 in blocks of 16 (9); 520 in blocks of 32 (10).  Alone at most one CTA
# per block and head to an SM, in the batch more
@pytest.mark.parametrize("K,V", [(64, 64), (32, 32), (16, 32)])
@pytest.mark.parametrize("T,H,B", [(128, 4, 40), (9001, 8, 4), (64 * 300 - 3, 6, 3), (64 * 520, 8, 2)])
def test_alone_batched_packed_and_by_head(K, V, T, H, B):
    L = 18                                            # packed: up to 2048 chunks, twice what the 64 x 64 pass on tcgen05 carries
    rows = [_draw(10 * T + i, T, H, K, V, L) for i in range(B)]
    batch = [torch.cat(t) for t in zip(*rows)]
    cu = torch.arange(B + 1, dtype=torch.int64, device="cuda") * T
    packed = [t.reshape(1, B * T, *t.shape[2:]) for t in batch]
    for op in (_hier, _plain):
        together, _ = op(batch)
        as_packed = op(packed, cu)[0].view_as(together)
        assert torch.equal(together, as_packed)
        for i in (0, B - 1):
            alone, _ = op(rows[i])
            assert torch.equal(alone[0], together[i])
            assert torch.equal(op(rows[i], torch.tensor([0, T], device="cuda"))[0], alone)
        for a, b in ((0, 1), (1, H)):
            assert torch.equal(op(_heads(rows[0], a, b))[0], together[:1, :, a:b])
    lampa_b200.check_status(torch.device("cuda:0"))


def test_short_and_long_sequences_packed():
    """64 x 64 heads: a sequence of more than 65,536 tokens beside shorter ones, an empty one among them."""
    H, L, lens = 2, 18, [700, 65600, 0, 33280, 65536, 1]
    rows = [_draw(7 + i, n, H, 64, 64, L) for i, n in enumerate(lens)]
    cu = torch.tensor([0] + lens).cumsum(0)
    together, _ = _hier([torch.cat(t, dim=1) for t in zip(*rows)], cu.cuda())
    for i, n in enumerate(lens):
        if n > 0:
            assert torch.equal(_hier(rows[i])[0], together[:, cu[i] : cu[i + 1]]), n
    lampa_b200.check_status(torch.device("cuda:0"))


def test_model_event_alone_and_in_a_batch():
    from lampa_b200 import synth
    from lampa_b200.model import LSHGatedDelta
    lengths = [9001, 700, 20003, 1, 6007, 12000]
    hits = [synth.detector_hits(50 + i, n).cuda() for i, n in enumerate(lengths)]
    torch.manual_seed(1)
    m = LSHGatedDelta(max_hits_per_event=60000).cuda()
    cu = torch.zeros(len(lengths) + 1, dtype=torch.int64)
    cu[1:] = torch.tensor(lengths).cumsum(0)
    full = m(torch.cat(hits), cu.cuda())
    for i, n in enumerate(lengths):
        assert torch.equal(m(hits[i], torch.tensor([0, n], device="cuda")), full[cu[i] : cu[i + 1]]), n


# tails of nothing, of either form of the tail kernel (16 tokens and more at once at K = 64, 48 at smaller heads) and of 63; a prompt
# alone has a CTA per eight state columns, the batches have CTAs that work through several
@pytest.mark.parametrize("K,V,H,B", [(64, 64, 8, 3), (64, 64, 8, 24), (32, 32, 8, 6), (16, 32, 8, 40), (64, 64, 2, 40)])
@pytest.mark.parametrize("T", [57, 128, 143, 144, 191, 320 + 31])
def test_prompts_alone_and_in_a_batch(K, V, H, B, T):
    L = 12
    rows = [_draw(10 * T + i, T, H, K, V, L) for i in range(B)]
    o, st = _hier([torch.cat(t) for t in zip(*rows)], state=True)
    for i in (0, B - 1):
        oi, si = _hier(rows[i], state=True)
        assert torch.equal(oi[0], o[i]) and torch.equal(si.states[0], st.states[i])
    for a, b in ((0, 1), (1, H)):
        oh, sh = _hier(_heads(rows[0], a, b), state=True)
        assert torch.equal(oh[0], o[0, :, a:b]) and torch.equal(sh.states[0], st.states[0, a:b])
    lampa_b200.check_status(torch.device("cuda:0"))
