"""Kernel variants picked by a rule on sizes, at the sizes where the rule or a tile edge lies."""
import numpy as np
import pytest

from mummu_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I,E,K", [(256, 128, 8, 2), (260, 132, 5, 3), (64, 36, 4, 1), (1028, 68, 3, 2)])
def test_f32_few_rows_same_bits_as_the_tile_kernel(cuda_lib, H, I, E, K):
    """f32 weights: the streaming kernel (up to 16 rows per expert on average) and the tile kernel sum in the
    same order, so a token has the same bits whichever ran; widths that are no multiple of a tile."""
    from mummu_b200 import moe
    L = cuda_lib
    T = 40 * E // K                                  # 40 rows per expert: the tile kernel
    router, gate, up, down, x = synth.moe_layer(H, I, E, T, cfg_seed=3)
    m = moe.SparseMoeConfig(H, I, E, K).init(device=0, act_dtype=L.F32, weight_dtype=L.F32)
    m.set_router(router)
    m.set_banks(gate, up, down)
    whole = m.forward(x, K, True)
    want, _, _ = O.moe_forward(x[:9], router, gate, up, down, K, True)
    assert np.abs(whole[:9] - want).max() <= 1e-5 * np.abs(want).max()
    for t in (1, 4 * E // K, 4 * E // K + 1, 16 * E // K):
        assert np.array_equal(m.forward(x[:t], K, True).view(np.uint32), whole[:t].view(np.uint32)), t
    m.close()


@pytest.mark.parametrize("dtype", ["bf16", "f16", "q4_k"])
@pytest.mark.parametrize("H,I,E,K,T,skew", [(256, 256, 2, 1, 1537, 0.0), (512, 256, 4, 2, 1600, 0.0), (256, 512, 8, 2, 3100, 1.0)])
def test_pair_gemm_against_the_single_cta_gemm(cuda_lib, dtype, H, I, E, K, T, skew):
    """From 768 rows per expert on average pairs of CTAs run the 16-bit GEMMs: ragged and empty segments, rows past
    the end of a 256-row tile.  Both kernels add the same products in the same order; the bound is one rounding of
    the 16-bit intermediate and output either way (2^-8 for bf16, 2^-10 for f16) on the largest value."""
    import torch
    from mummu_b200 import moe
    L = cuda_lib
    act = L.BF16 if dtype == "bf16" else L.F16
    tdt = torch.bfloat16 if dtype == "bf16" else torch.float16
    g = torch.Generator(device="cuda").manual_seed(5)
    m = moe.SparseMoeConfig(H, I, E, K).init(device=0, act_dtype=act, weight_dtype=L.Q4_K if dtype == "q4_k" else act)
    bias = synth.zipf_router_bias(E, 3.0) if skew else None
    m.set_router((torch.randn(H, E, generator=g, device="cuda") * 0.1).cpu().numpy(), bias=bias)
    for which, shape in ((L.BANK_GATE, (E, I, H)), (L.BANK_UP, (E, I, H)), (L.BANK_DOWN, (E, H, I))):
        w = torch.randn(shape, generator=g, device="cuda") * 0.05
        m.set_bank(which, moe.q4k_quantize_device(w) if dtype == "q4_k" else w.to(tdt))
    x = torch.randn(T, H, generator=g, device="cuda").to(tdt)
    whole = m.forward(x, K, False)
    part = 768 * E // K - 1                           # one token short of the rule
    single = m.forward(x[:part].contiguous(), K, False)
    m.sync()
    top = single.float().abs().max().item()
    assert (whole[:part].float() - single.float()).abs().max().item() <= (2.0 ** -8 if dtype == "bf16" else 2.0 ** -10) * top
    assert torch.isfinite(whole.float()).all()
    m.close()


@pytest.mark.parametrize("kv_heads", [4, 2])
def test_static_step_over_split_keys_equals_the_growing_cache_step(cuda_lib, kv_heads):
    """Sequences of very different lengths in one step: the key splits follow each sequence's own length (some
    of them without a key), and the partials fold to the step of the growing-cache path.  Both round the same
    16-bit activations; 2e-2 of the largest logit is the bar the model tests use."""
    import torch
    from mummu_b200 import _lib as L
    from mummu_b200.olmoe import OlmoeConfig, OlmoeDecoder
    cfg = OlmoeConfig(vocab_size=256, hidden_size=256, intermediate_size=256, num_hidden_layers=2,
                      num_attention_heads=4, num_key_value_heads=kv_heads, num_experts=4, num_experts_per_tok=2)
    lengths = [1, 31, 300, 639]
    B, ctx = len(lengths), 640
    dec = OlmoeDecoder(cfg, device=0, expert_dtype=L.Q4_K, max_batch=B, max_ctx=ctx)
    if kv_heads != 4:                                  # random_init draws square k / v projections
        dec.random_init(seed=1)
        for lay in dec.layers:
            n = kv_heads * cfg.head_dim
            lay.update(k=lay["k"][:n].contiguous(), v=lay["v"][:n].contiguous(), k_norm=lay["k_norm"][:n].contiguous())
    else:
        dec.random_init(seed=1)
    dec.embed.mul_(50.0)
    g = torch.Generator(device="cuda").manual_seed(2)
    dec.k_cache.normal_(generator=g)
    dec.v_cache.normal_(generator=g)
    ids = torch.randint(0, cfg.vocab_size, (B, 1), generator=g, device="cuda")
    state = dec.static_state(B, ctx)
    for b in range(B):
        dec.seed_static(state, b, lengths[b])
    got = dec.forward_static(ids.to(torch.int32), torch.tensor(lengths, dtype=torch.int32, device="cuda"), state, ctx).clone()
    for b in range(B):
        dec.k_cache[:, 0].copy_(dec.k_cache[:, b].clone())
        dec.v_cache[:, 0].copy_(dec.v_cache[:, b].clone())
        want = dec.forward(ids[b:b + 1], lengths[b])
        assert (got[b] - want[0]).abs().max().item() <= 2e-2 * want.abs().max().item(), lengths[b]
        assert state.argmax[b].item() == got[b].argmax().item()
    state.close()
    dec.close()
