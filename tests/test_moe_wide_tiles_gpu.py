"""Routed FFNs at the edges of their routes: one-launch routing (to 128 rows), grouped tiles on pairs of CTAs (128 wide, whole pairs of
feature tiles), experts without rows, tokens whose experts another rank holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,E,k,hidden,inter", [
    (127, 128, 8, 512, 256), (128, 256, 8, 256, 256), (129, 128, 8, 512, 256),      # one launch or several
    (300, 4, 2, 512, 256), (700, 8, 2, 512, 768), (2100, 8, 3, 1024, 256),          # pairs of CTAs
    (700, 8, 2, 384, 256), (700, 8, 2, 512, 384),                                   # an odd number of feature tiles in one product
])
@pytest.mark.parametrize("half", [False, True])
def test_against_dense_loops(rows, E, k, hidden, inter, half):
    from crosspool_b200.models.config import ModelConfig
    from crosspool_b200.models.reference import moe_ffn
    from crosspool_b200.models.weights import FfnLayerWeights, random_ffn_layer
    from crosspool_b200.ops import gemm, moe
    from crosspool_b200.testing import assert_ffn_close

    cfg = ModelConfig(name="t", architecture="Qwen3MoeForCausalLM", hidden_size=hidden, num_layers=1, num_q_heads=4, num_kv_heads=2, head_dim=64,
                      intermediate_size=inter, vocab_size=128, num_experts=E, num_experts_per_tok=k, moe_intermediate_size=inter)
    w = random_ffn_layer(cfg, 0, seed=rows, device="cuda", dtype=torch.bfloat16)
    x = (torch.randn(rows, hidden, device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows)) * 0.5).bfloat16()
    ref = moe_ffn(x, w, cfg)
    if half:       # two ranks' partial sums
        y = torch.zeros(rows, hidden, device="cuda")
        for lo, hi in ((0, E // 2), (E // 2, E)):
            part = FfnLayerWeights(w.gate_up[lo:hi].contiguous(), w.down[lo:hi].contiguous(), w.router)
            y += moe.moe_forward(x, part, cfg, expert_range=(lo, hi)).float()
    else:
        y = moe.moe_forward(x, w, cfg).float()
    gemm.check_status(x.device)
    assert_ffn_close(y, ref.float())
