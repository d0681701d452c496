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
