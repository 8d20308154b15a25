"""Decode sessions on the chain of packed linears (bf16 tables, one GPU): against the model's own parts in 64 bits."""
import pytest
import torch

from nativebit_b200 import generate as G

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _model(seed=0, layers=1, **kw):
    cfg = G.ModelConfig(**{**dict(vocab_size=512, n_layers=layers, n_embd=256, n_head=4, ffn_hidden=512, context_len=64), **kw})
    return G.PackedGPT.random_init(cfg, seed=seed)


@pytest.mark.parametrize("size", [1e-3, 1.0, 1e5])
@pytest.mark.parametrize("batch", [9, 16, 40])
def test_rows_of_any_size_keep_their_bits(built_lib, batch, size):
    """A norm takes the size out of its rows: q | k | v of rows of 1e-3 and of 1e5 is as exact as that of rows around one."""
    model = _model()
    model.embedding.copy_(size * torch.randn(512, 256, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1)))
    blk = model.blocks[0]
    blk.ln1.copy_(1 + 0.1 * torch.randn(256, device=DEV, generator=torch.Generator(device=DEV).manual_seed(2)))
    s = model.session(batch)
    assert s.chain
    s.token.copy_(torch.randint(0, 512, (batch, 1), device=DEV))
    tokens = s.token[:, 0].clone()
    s.step()
    s.check()
    x = model.embedding[tokens].double()
    h = x / torch.sqrt((x * x).mean(-1, keepdim=True) + model.config.norm_eps) * blk.ln1.double()
    want = h @ blk.qkv.dequantized_weight().double().T
    # 22-bit operands, sums in fp32: a few 2^-22 of the norm
    assert (s.bqkv.double() - want).norm() <= 2e-6 * want.norm()
