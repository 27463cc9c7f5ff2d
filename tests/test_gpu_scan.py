"""The scan's kernels on either side of the rules that choose their shape (compose: S and P together or in CTAs of their own;
level: all slabs of a head or one per CTA), against the token recurrence, and outputs in every type that has its own store."""
import numpy as np
import pytest
import torch

from oracle import oracle
from tests.util import assert_close_bf16, to_np

pytestmark = pytest.mark.gpu


def _call(inp, levels, cu=None, dt=torch.bfloat16):
    import lampa_b200
    d = {k: v.cuda() for k, v in inp.items()}
    q, k, v = (d[n].to(dt) for n in ("q", "k", "v"))
    if levels:
        o, _ = lampa_b200.chunk_h_gated_delta_rule(q, k, v, d["g"], d["lam"], d["beta"], cu_seqlens=cu, use_qk_l2norm_in_kernel=True)
        return to_np(o[0]), None
    o, ht = lampa_b200.chunk_gated_delta_rule(q, k, v, d["g"], d["beta"], cu_seqlens=cu, output_final_state=True, use_qk_l2norm_in_kernel=True)
    return to_np(o[0]), to_np(ht)


def _ref(inp, levels, cu=None):
    a = [to_np(inp[n][0]) for n in ("q", "k", "v", "g", "beta")]
    if levels:
        return oracle.hgdn(*a, to_np(inp["lam"][0]), cu_seqlens=cu, use_l2norm=True)[0], None
    return oracle.gdn_plain(*a, cu_seqlens=cu, use_l2norm=True)


# blocks x heads on either side of 148 (the SMs of a B200): 2 x 32, 6 x 25 and 5 x 30 blocks; one block; a last block of one ragged chunk
@pytest.mark.parametrize("K,V", [(64, 64), (32, 32), (16, 32)])
@pytest.mark.parametrize("T,H", [(512, 1), (513, 2), (64 * 256, 2), (64 * 24 * 8 + 1, 6), (64 * 30 * 16 - 5, 5)])
def test_plain_shapes(K, V, T, H):
    from lampa_b200 import synth
    inp = synth.gdn_inputs(31, T, H, K, V, g_shift=-4.0)
    o, ht = _call(inp, 0)
    ro, rh = _ref(inp, 0)
    assert_close_bf16(o, ro, f"o {T}x{H}")
    assert_close_bf16(ht, rh, f"state {T}x{H}")


@pytest.mark.parametrize("K,V", [(64, 64), (32, 32), (16, 32)])
@pytest.mark.parametrize("n,H", [(36, 2), (38, 2), (80, 1)])
def test_many_short_sequences(K, V, n, H):
    """One CTA per slab up to 296 slabs (sequences x heads x levels x V / 16), whole heads beyond; some sequences are empty."""
    from lampa_b200 import synth
    rng = np.random.default_rng(5)
    lens = rng.integers(0, 700, n)
    lens[3] = 0
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    inp = synth.gdn_inputs(32, int(cu[-1]), H, K, V, L=12, g_shift=-3.0)
    ro, rh = _ref(inp, 0, cu)
    cu_dev = torch.from_numpy(cu).cuda()
    o, ht = _call(inp, 0, cu_dev)
    assert_close_bf16(o, ro, "o")
    assert_close_bf16(ht, rh, "state")
    assert_close_bf16(_call(inp, 12, cu_dev)[0], _ref(inp, 12, cu)[0], "o, levels")


@pytest.mark.parametrize("K,V", [(64, 64), (16, 32)])
@pytest.mark.parametrize("T", [1, 63, 64 * 9 + 1])
def test_fp16_rows(K, V, T):
    from lampa_b200 import synth
    inp = synth.gdn_inputs(33, T, 3, K, V, g_shift=-3.0)
    o, _ = _call(inp, 0, dt=torch.float16)
    assert_close_bf16(o, _ref(inp, 0)[0], "o fp16")


# blocks x heads at most 148 and above it: levels shared out over warps, or five to a warp; a sequence of one block, a ragged one,
# blocks of 8, 16 and 32 chunks
@pytest.mark.parametrize("K,V", [(32, 32), (16, 32)])
@pytest.mark.parametrize("T,H", [(64 * 3, 1), (64 * 8 * 9 + 5, 3), (64 * 256, 4), (64 * 300, 6), (64 * 304, 8), (64 * 520, 2)])
def test_levels_by_warp(K, V, T, H):
    from lampa_b200 import synth
    inp = synth.gdn_inputs(34, T, H, K, V, L=18, g_shift=-4.0)
    assert_close_bf16(_call(inp, 18)[0], _ref(inp, 18)[0], f"o, levels {T}x{H}")
