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
