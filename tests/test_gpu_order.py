"""What a launch may read before the one in front of it has ended: weights that were written a moment ago, by another stream, or
under capture."""
import pytest
import torch

from nativebit_b200 import PackedLinear, ops
from nativebit_b200 import generate as G

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_a_table_dequantised_a_launch_ago_is_what_the_head_reads(built_lib):
    """The LM head asks for rows of its table ahead of its dependency wait: nb_dequant may not let it start early."""
    v, c = 16384, 2560
    g = torch.Generator(device=DEV).manual_seed(0)
    packed = ops.pack(torch.randint(0, 8, (v * c,), dtype=torch.uint8, device=DEV, generator=g), 3)
    cb = torch.randn(v * c // 128, 8, device=DEV, generator=g).half()
    x = torch.randn(1, c, device=DEV, generator=g)

    def head(table):
        logits, tok = torch.empty(1, v, device=DEV), torch.zeros(1, 1, dtype=torch.long, device=DEV)
        ops.lm_head(x, None, None, 1e-6, table, 30.0, logits, tok, None)
        return logits

    table = ops.dequant(packed, cb, 3, 128, (v, c), torch.bfloat16)
    torch.cuda.synchronize()
    want = head(table)
    for _ in range(5):
        table.fill_(float("nan"))
        del table                                     # the next one takes its memory
        table = ops.dequant(packed, cb, 3, 128, (v, c), torch.bfloat16)
        assert torch.equal(head(table), want)


def _weights(n, k, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (ops.pack(torch.randint(0, 8, (n * k,), dtype=torch.uint8, device=DEV, generator=g), 3),
            torch.randn(n * k // 128, 8, device=DEV, generator=g).half())


@pytest.mark.parametrize("rows,n,k", [(4, 6912, 2560), (40, 1024, 1024), (100, 6912, 2560)])
def test_a_linear_that_several_streams_ask_first(built_lib, rows, n, k):
    """The first calls, one behind the other on two streams, then on both after other weights were loaded."""
    torch.cuda.synchronize()
    w, other = _weights(n, k, 1), _weights(n, k, 2)
    x = torch.randn(rows, k, device=DEV, generator=torch.Generator(device=DEV).manual_seed(3))
    streams = [torch.cuda.Stream() for _ in range(2)]
    for load in (None, other):
        want = PackedLinear(*(load or w), n, k)(x)
        if load is None:
            lin = PackedLinear(w[0].clone(), w[1].clone(), n, k)
        else:
            lin.load_state_dict({"packed_indices": load[0], "codebook": load[1]})
        torch.cuda.synchronize()
        got = []
        for s in streams:
            with torch.cuda.stream(s):
                got.append(lin(x))
        torch.cuda.synchronize()
        assert all(torch.equal(y, want) for y in got)


@pytest.mark.parametrize("rows", [4, 40, 100])
def test_a_linear_whose_first_call_of_many_rows_is_captured(built_lib, rows):
    """The graph that would have to make the copy leaves none behind: calls before and after its replay are right, and so is it."""
    n, k = 2560, 1024
    w = _weights(n, k, 4)
    g = torch.Generator(device=DEV).manual_seed(5)
    x, big = torch.randn(rows, k, device=DEV, generator=g), torch.randn(300, k, device=DEV, generator=g)
    want = PackedLinear(*w, n, k)(x).double()
    lin = PackedLinear(*w, n, k)
    lin(x[:1])
    PackedLinear(*w, n, k)(big.repeat(4, 1))                  # the workspaces are there
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = lin(x)
    assert not lin._copied_now() or rows <= 16
    eager = lin(x)
    graph.replay()
    for got in (y, eager, lin(x)):                            # sums of other kernels in fp32: a few 2^-24 of the norm
        assert (got.double() - want).norm() <= 2e-6 * want.norm()


def _run(session, prompt, steps=3):
    """The logits of a prompt and of the steps behind it over given tokens."""
    out = [session.prefill(prompt).clone()]
    for _ in range(steps):
        session.token.fill_(7)
        session.step()
        out.append(session.logits.clone())
    return torch.stack(out)


def _two_models():
    cfg = G.ModelConfig(vocab_size=512, n_layers=2, n_embd=256, n_head=4, ffn_hidden=512, context_len=64)
    return G.PackedGPT.random_init(cfg, seed=0), G.PackedGPT.random_init(cfg, seed=1)


@pytest.mark.parametrize("batch", [1, 4, 12, 40])
def test_sessions_follow_other_weights_from_the_next_prompt_on(built_lib, batch):
    """After other weights were loaded under captured prompts and steps, or took the place of the tensors, a prompt of a known and one
    of a new length and the steps behind them are those of a session made with these weights."""
    model, other = _two_models()
    third = G.PackedGPT.random_init(model.config, seed=2)
    g = torch.Generator(device=DEV).manual_seed(6)
    prompts = [torch.randint(0, 512, (batch, t), device=DEV, generator=g) for t in (20, 20, 33)]
    session = model.session(batch)
    _run(session, prompts[0])
    model.load_state_dict(other.state_dict())
    for prompt in prompts[1:]:
        assert torch.equal(_run(session, prompt), _run(other.session(batch), prompt))
    for a, b in zip(model.blocks, third.blocks):
        for name in ("qkv", "out_proj", "gate_up", "down"):
            getattr(a, name).packed_indices, getattr(a, name).codebook = getattr(b, name).packed_indices, getattr(b, name).codebook
    model.embedding.copy_(third.embedding)
    for prompt in prompts[1:]:
        assert torch.equal(_run(session, prompt), _run(third.session(batch), prompt))
    a, b = other.session(batch), third.session(batch)       # in the middle of a sequence: the next step
    for s in (a, b):
        _run(s, prompts[0])
    for (k, v, _), (k2, v2, _) in zip(a.caches, b.caches):
        k2.copy_(k), v2.copy_(v)
    other.load_state_dict(third.state_dict())
    for _ in range(2):
        for s in (a, b):
            s.token.fill_(5)
            s.step()
        assert torch.equal(a.logits, b.logits)
    for a, b in zip(model.blocks, third.blocks):
        assert torch.equal(a.gate_up.stream_weight(1), b.gate_up.stream_weight(1)) and torch.equal(a.qkv.stream_weight(), b.qkv.stream_weight())


@pytest.mark.parametrize("batch", [9, 16])
def test_captured_steps_over_the_packed_bytes_follow_what_is_written_to_them(built_lib, batch):
    """Nine to sixteen sequences: a step that was captured before other weights were written in place, counted or not, multiplies them."""
    model, other = _two_models()
    session = model.session(batch)
    assert session.chain_packed
    prompt = torch.randint(0, 512, (batch, 1), device=DEV)
    _run(session, prompt)
    for blk, src in zip(model.blocks, other.blocks):
        for name in ("qkv", "out_proj", "gate_up", "down"):
            getattr(blk, name).packed_indices.data.copy_(getattr(src, name).packed_indices)
            getattr(blk, name).codebook.data.copy_(getattr(src, name).codebook)
    torch.cuda.synchronize()
    want = other.session(batch)
    for s in (session, want):
        s.reset()
        s.token.fill_(3)
        for k, v, _ in s.caches:
            k.zero_(), v.zero_()
    model.embedding.copy_(other.embedding)
    for _ in range(3):
        session.step(), want.step()
        assert torch.equal(session.logits, want.logits)
    assert not any("_wstream" in lin.__dict__ for blk in model.blocks for lin in (blk.qkv, blk.out_proj, blk.gate_up, blk.down))
