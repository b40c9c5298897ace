"""Activation recomputation on the kernels, some of which work in place: the gradients of a run that keeps everything."""
import pytest
import torch

from primus_b200.models.config import TransformerConfig
from primus_b200.models.gpt import GPTModel
from primus_b200.parallel import state as ps

pytestmark = pytest.mark.gpu


def _grads(**kw):
    cfg = TransformerConfig(num_layers=2, hidden_size=256, ffn_hidden_size=512, num_attention_heads=4, num_query_groups=2,
                            vocab_size=512, make_vocab_size_divisible_by=64, seq_length=128, **kw)
    ps.destroy_model_parallel()
    ps.initialize_model_parallel()
    torch.manual_seed(3)
    m = GPTModel(cfg, "cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    tok, lab = (torch.randint(0, 512, (2, 128), device="cuda", generator=g) for _ in range(2))
    loss = m(tok, lab, loss_weights=torch.full((2, 128), 1.0 / 256, device="cuda"))
    loss.backward()
    grads = {n: (p.grad if p.grad is not None else p.main_grad).detach().clone() for n, p in m.named_parameters()
             if p.grad is not None or getattr(p, "main_grad", None) is not None}
    ps.destroy_model_parallel()
    return float(loss.detach()), grads


@pytest.mark.parametrize("qk_layernorm", [False, True])
@pytest.mark.parametrize("kw", [dict(recompute_granularity="full", recompute_method="uniform", recompute_num_layers=1),
                                dict(recompute_granularity="selective"),
                                dict(recompute_granularity="selective", recompute_modules=["core_attn", "mlp"])])
def test_recompute_gives_the_same_gradients(kw, qk_layernorm):
    loss, want = _grads(qk_layernorm=qk_layernorm)
    again, got = _grads(qk_layernorm=qk_layernorm, **kw)
    assert loss == again and got.keys() == want.keys()
    for n, t in want.items():
        if "embedding" in n:                # (summed by atomics in fp32, then rounded)
            assert (got[n].float() - t.float()).norm() <= 2.0 ** -9 * t.float().norm(), n
        else:
            assert torch.equal(got[n], t), n
