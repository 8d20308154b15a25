"""Decode sessions on the chain of packed linears (bf16 tables, one GPU): against the model's own parts in 64 bits."""
import os

import numpy as np
import pytest
import torch

from nativebit_b200 import generate as G
from oracle import nb_model_oracle as mo

pytestmark = pytest.mark.gpu
DEV = "cuda"
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "reference_model.npz")


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


@pytest.mark.parametrize("batch", [1, 2, 8, 9, 16, 32])
def test_steps_of_the_reference_model_against_the_dense_oracle(built_lib, batch):
    """The reference's own packed layers under a bf16 table: prompts that differ from sequence to sequence and given tokens behind them,
    captured, against the dense oracle in fp32."""
    gm = np.load(GOLDEN)
    v, layers, c, heads, ffn, ctx = (int(x) for x in gm["cfg"])
    cfg = G.ModelConfig(vocab_size=v, n_layers=layers, n_embd=c, n_head=heads, ffn_hidden=ffn, context_len=ctx)

    def cu(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    blocks = []
    for i in range(layers):
        full = {to: (cu(gm[f"p_{name}{i}"]), cu(gm[f"c_{name}{i}"])) for name, to in (("qkv", "qkv"), ("out", "out_proj"), ("gate", "gate"), ("up", "up"), ("down", "down"))}
        blocks.append(G.shard_block(cfg, full, torch.ones(c, device=DEV), torch.ones(c, device=DEV), 0, 1))
    table = torch.from_numpy(gm["embedding"]).bfloat16()
    model = G.PackedGPT(cfg, table.to(DEV), blocks, torch.ones(c, device=DEV))
    packed = {f"{n}{i}": (gm[f"p_{n}{i}"], gm[f"c_{n}{i}"], tuple(int(x) for x in gm[f"s_{n}{i}"])) for i in range(layers) for n in ("qkv", "out", "gate", "up", "down")}
    dense = mo.DenseModel(mo.dense_weights_from_packed(packed, table.float().numpy(), layers), layers, heads, ctx)
    caches = dense.init_cache(batch)
    g = torch.Generator().manual_seed(batch)
    prompt = torch.randint(0, v, (batch, gm["prompt"].shape[1]), generator=g)
    prompt[0] = torch.from_numpy(gm["prompt"])[0]
    s = model.session(batch, chain=True)
    want = dense.forward(prompt, caches)[:, -1]
    got = s.prefill(prompt.to(DEV)).cpu()
    for step in range(6):
        # fp32 sums in another order through every layer: the other routes' tests allow the same
        assert (got - want).abs().max() <= 1e-4 * want.abs().max(), step
        token = torch.randint(0, v, (batch, 1), generator=g)
        s.token.copy_(token)
        s.step()
        got, want = s.logits.cpu(), dense.forward(token, caches)[:, -1]
    s.check()


@pytest.mark.parametrize("batch", [2, 8, 9, 16, 20, 64])
def test_steps_on_the_chain_equal_the_other_kernels(built_lib, batch):
    """Against the same session without the chain: the same tokens, logits within the order of the sums; from a graph as eagerly."""
    model = _model(seed=5, layers=3, n_embd=512, ffn_hidden=1408)
    prompt = torch.randint(0, 512, (batch, 7), generator=torch.Generator().manual_seed(batch)).to(DEV)
    a, e, b = model.session(batch, chain=True), model.session(batch, chain=True, use_graph=False), model.session(batch, chain=False)
    assert a.chain and not b.chain and a.chain_packed == (9 <= batch <= 16)
    for s in (a, e, b):
        s.prefill(prompt)
    for _ in range(8):
        for s in (a, e, b):
            s.step()
        assert torch.equal(a.logits, e.logits) and torch.equal(a.token, b.token)
        assert (a.logits - b.logits).abs().max() <= 1e-4 * b.logits.abs().max()
    for s in (a, e, b):
        s.check()


@pytest.mark.parametrize("batch", [1, 4, 12, 40])
def test_nan_in_a_cache_reaches_the_logits_of_its_sequence(built_lib, batch):
    model = _model(layers=2)
    s = model.session(batch, chain=True)
    s.prefill(torch.randint(0, 512, (batch, 5), device=DEV))
    s.caches[0][1][batch - 1, 2, 1, 7] = float("nan")            # one value of one head
    s.step()
    nan = s.logits.isnan()
    assert bool(nan[batch - 1].all()) and not bool(nan[:batch - 1].any())


def test_a_chain_that_is_asked_for_and_cannot_be_is_refused(built_lib):
    model = _model()
    assert not model.session(2, chain=False).chain
    model.embedding = model.embedding.float()
    assert not model.session(2).chain
    with pytest.raises(RuntimeError, match="chain"):
        model.session(2, chain=True)
