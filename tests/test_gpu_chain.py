"""The decode chain's packed linears (nb_chain_linear, nb_chain_embed) against fp64 products of the oracle's dense weight."""
import numpy as np
import pytest
import torch

from nativebit_b200 import PackedLinear, ops
from nativebit_b200.stream import stream_pack
from oracle import nb_oracle as o

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _matrix(n, k, bits, seed, row_mode=0):
    packed, cb, _ = o.make_packed_linear(n, k, bits, seed=seed)
    w = stream_pack(torch.from_numpy(packed).to(DEV), torch.from_numpy(cb).to(DEV), bits, n, k, row_mode)
    return w, torch.from_numpy(o.dequant_packed(packed, cb.astype(np.float32), n, k, bits)).to(DEV).double()


def _terms(x):
    """(m, k) fp32 -> the layout of nb_chain_linear, written out from its description."""
    m, k = x.shape
    hi = x.clamp(-65504, 65504).half()
    lo = (x - hi.float()).half()
    out = torch.zeros(m, 2, k // 128, 4, 4, 8, dtype=torch.float16, device=DEV)      # row, term, block, segment, chunk, value
    for s, v in enumerate((hi, lo)):
        v = v.view(m, k // 128, 4, 4, 8)[..., [0, 2, 1, 3, 4, 6, 5, 7]]
        for t in range(4):
            for c in range(4):
                out[:, s, :, t, c ^ t ^ s] = v[:, :, t, c]
    return out.view(torch.uint8).reshape(-1)


def _values(terms, m, k):
    t = terms[:4 * m * k].view(torch.float16).view(m, 2, k // 128, 4, 4, 8).double()
    out = torch.zeros(m, k // 128, 4, 4, 8, dtype=torch.float64, device=DEV)
    for s in range(2):
        for seg in range(4):
            for c in range(4):
                out[:, :, seg, c] += t[:, s, :, seg, c ^ seg ^ s]
    return out[..., [0, 2, 1, 3, 4, 6, 5, 7]].view(m, k)


def _close(got, want, rel):
    assert torch.isfinite(got.double()).all()
    err = (got.double() - want).norm() / want.norm()
    assert err <= rel, float(err)


# fp32 sums of products of 22-bit activations and exact weights: a few 2^-22 of the norm (2.4e-7 each)
REL = 2e-6
SHAPES = [(16, 128, 1), (40, 128, 3), (256, 384, 1), (2560, 2560, 1), (2560, 6912, 1), (2560, 6912, 2), (1000, 1024, 4), (7680, 2560, 5),
          (2560, 6912, 8), (5632, 2048, 8), (512, 2560, 9), (2560, 6912, 16), (2560, 2560, 17), (3072, 1024, 32), (30000, 256, 1)]


@pytest.mark.parametrize("n,k,m", SHAPES)
@pytest.mark.parametrize("bits", [2, 3, 4])
def test_chain_linear_stores_the_product(built_lib, n, k, m, bits):
    w, dense = _matrix(n, k, bits, seed=n + k + m)
    g = torch.Generator(device=DEV).manual_seed(m)
    x = torch.randn(m, k, device=DEV, generator=g)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = x.double() @ dense.T
    ran = 0
    for split in (0, 1, 2, 4, 8):
        y = torch.full((m, n), float("nan"), device=DEV)
        try:
            ops.chain_linear(ops.CHAIN_STORE, w, bits, m, n, k, _terms(x), status, y=y, split=split)
        except RuntimeError as e:
            assert split and "shape" in str(e)            # more CTAs than k-blocks, or the activations do not fit
            continue
        ran += 1
        _close(y, want, REL)
        again = torch.empty_like(y)
        ops.chain_linear(ops.CHAIN_STORE, w, bits, m, n, k, _terms(x), status, y=again, split=split)
        assert torch.equal(y, again)
    assert ran >= 2 and int(status.item()) == 0


@pytest.mark.parametrize("m,c,f", [(1, 256, 512), (3, 1024, 2816), (8, 2560, 6912), (20, 384, 640)])
def test_chain_carries_norms_and_residuals(built_lib, m, c, f):
    """embedding -> gate | up -> down -> a linear of the normed result."""
    bits, eps = 3, 1e-6
    g = torch.Generator(device=DEV).manual_seed(c)
    table = torch.randn(50, c, device=DEV, generator=g).bfloat16()
    token = torch.randint(0, 50, (m, 1), device=DEV, generator=g)
    w1, w2 = (1 + 0.1 * torch.randn(c, device=DEV, generator=g) for _ in range(2))
    gu, gu_dense = _matrix(2 * f, c, bits, 1, row_mode=1)
    down, down_dense = _matrix(c, f, bits, 2)
    last, last_dense = _matrix(400, c, bits, 3)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    x, sq = torch.empty(m, c, device=DEV), torch.empty(m, c // 16, device=DEV)
    cx, ch = ops.chain_terms(m, c, DEV), ops.chain_terms(m, f, DEV)
    ops.chain_embed(table, token, w1, x, cx, sq)
    emb = table[token[:, 0]].double()
    assert torch.equal(x.double(), emb)
    _close(_values(cx, m, c), emb * w1.double(), REL)
    _close(sq.double().sum(1), (emb * emb).sum(1), REL)

    def rms(v, w):
        return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps) * w.double()
    ops.chain_linear(ops.CHAIN_SWIGLU, gu, bits, m, 2 * f, c, cx, status, sq=sq, eps=eps, y_terms=ch)
    z = rms(emb, w1) @ gu_dense.T
    h = torch.nn.functional.silu(z[:, :f]) * z[:, f:]
    _close(_values(ch, m, f), h, 4 * REL)                 # + the fast exponential
    ops.chain_linear(ops.CHAIN_RESIDUAL, down, bits, m, c, f, ch, status, residual=x, y_terms=cx, next_weight=w2, sq_out=sq)
    r = emb + h @ down_dense.T
    _close(x, r, 4 * REL)
    _close(_values(cx, m, c), r * w2.double(), 4 * REL)
    y = torch.empty(m, 400, device=DEV)
    ops.chain_linear(ops.CHAIN_STORE, last, bits, m, 400, c, cx, status, sq=sq, eps=eps, y=y)
    _close(y, rms(r, w2) @ last_dense.T, 8 * REL)
    before = x.clone()
    ops.chain_linear(ops.CHAIN_RESIDUAL, down, bits, m, c, f, ch, status, residual=x)          # nothing behind it
    _close(x, before.double() + h @ down_dense.T, 4 * REL)
    assert int(status.item()) == 0


@pytest.mark.parametrize("n,k,m", [(16, 128, 1), (1000, 1024, 9), (2560, 6912, 16), (5632, 2048, 11), (333, 2560, 13), (4096, 256, 33)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits", [2, 3, 4])
def test_chain_rows_takes_plain_activations(built_lib, n, k, m, dtype, bits):
    w, dense = _matrix(n, k, bits, seed=n + m)
    x = torch.randn(m, k, device=DEV, generator=torch.Generator(device=DEV).manual_seed(k)).to(dtype)
    want = x.double() @ dense.T
    for ordered in (True, False):
        y = ops.chain_rows(x, w, bits, n, k, ordered=ordered, out=torch.full((m, n), float("nan"), dtype=torch.float32, device=DEV))
        _close(y, want, REL)
    y = ops.chain_rows(x, w, bits, n, k)
    assert y.dtype == dtype
    # a rounding of the result to nearest is at most half an ulp (2^-11, 2^-8) of each value
    _close(y, want, {torch.float32: REL, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype])


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 1e5])
def test_what_is_no_number_reaches_the_products_behind(built_lib, value):
    """gate | up -> down and attention -> out_proj hand their rows over as terms: NaN arrives in every output of its row, what fp16
    does not hold arrives as the largest two terms, and other rows are as they were."""
    m, c, f, bits = 3, 256, 512, 3
    g = torch.Generator(device=DEV).manual_seed(5)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    gu, gu_dense = _matrix(2 * f, c, bits, 1, row_mode=1)
    down, dense = _matrix(c, f, bits, 2)
    torch.cuda.synchronize()
    x = torch.randn(m, c, device=DEV, generator=g)
    x[1, 5] = value if value != value else 60000.0
    h = ops.chain_terms(m, f, DEV)
    ops.chain_linear(ops.CHAIN_SWIGLU, gu, bits, m, 2 * f, c, _terms(x), status, y_terms=h)
    y = torch.zeros(m, c, device=DEV)
    ops.chain_linear(ops.CHAIN_RESIDUAL, down, bits, m, c, f, h, status, residual=y)
    z = x.double() @ gu_dense.T
    want = (torch.nn.functional.silu(z[:, :f]) * z[:, f:]).clamp(-131008, 131008) @ dense.T
    assert torch.equal(y.isnan(), torch.tensor([False, value != value, False], device=DEV)[:, None].expand(m, c))
    _close(y[[0, 2]], want[[0, 2]], 4 * REL)
    if value == value:                                   # beyond 65504 the second term is up to 65504 itself, with an error of up to 16
        _close(y[1], want[1], 2.0 ** -12)

    heads, hd, ctx = 2, 64, 16                           # 128 columns of attention in front of an out_proj
    out, out_dense = _matrix(256, heads * hd, bits, 3)
    torch.cuda.synchronize()
    k, v = (torch.randn(m, heads, ctx, hd, device=DEV, generator=g) for _ in range(2))
    v[1, :, 2] = value
    cos2, sin2 = torch.ones(ctx, hd, device=DEV), torch.zeros(ctx, hd, device=DEV)
    qkv, pos = torch.randn(m, 3 * heads * hd, device=DEV, generator=g), torch.tensor([7], device=DEV)
    terms, plain = ops.chain_terms(m, heads * hd, DEV), torch.zeros(m, heads * hd, device=DEV)
    ops.decode_attention_rope(qkv, cos2, sin2, pos, k, v, plain, 0)
    ops.decode_attention_terms(qkv, cos2, sin2, pos, k, v, terms, heads * hd, 0)
    y = torch.zeros(m, 256, device=DEV)
    ops.chain_linear(ops.CHAIN_RESIDUAL, out, bits, m, 256, heads * hd, terms, status, residual=y)
    assert torch.equal(y.isnan(), plain.isnan().any(1, keepdim=True).expand(m, 256))
    _close(y[[0, 2]], plain[[0, 2]].double() @ out_dense.T, REL)
    if value == value:
        _close(y[1], plain[1].double().clamp(-131008, 131008) @ out_dense.T, 2.0 ** -12)


@pytest.mark.parametrize("n,k,m", [(16, 128, 2), (1000, 1024, 9), (2560, 6912, 16), (2560, 6912, 2), (5632, 2048, 11), (333, 2560, 13), (4096, 256, 33), (90000, 128, 16)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits", [2, 3, 4])
def test_chain_rows_over_the_packed_bytes(built_lib, n, k, m, dtype, bits):
    """The packed matrix itself in place of its stream-layout copy; codebooks of either type."""
    packed, cb, _ = o.make_packed_linear(n, k, bits, seed=n + m)
    dense = torch.from_numpy(o.dequant_packed(packed, cb.astype(np.float32), n, k, bits)).to(DEV).double()
    p, cb = torch.from_numpy(packed).to(DEV), torch.from_numpy(cb).to(DEV)
    x = torch.randn(m, k, device=DEV, generator=torch.Generator(device=DEV).manual_seed(k)).to(dtype)
    want = x.double() @ dense.T
    for codebook in (cb, cb.float()):
        for ordered in (True, False):
            y = ops.chain_rows(x, p, bits, n, k, ordered=ordered, out=torch.full((m, n), float("nan"), dtype=torch.float32, device=DEV), codebook=codebook)
            _close(y, want, REL)
            assert torch.equal(y, ops.chain_rows(x, p, bits, n, k, out=torch.empty_like(y), codebook=codebook))
    y = ops.chain_rows(x, p, bits, n, k, codebook=cb)
    assert y.dtype == dtype
    _close(y, want, {torch.float32: REL, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype])
    with pytest.raises(RuntimeError):
        ops.chain_rows(x, p[:-16], bits, n, k, codebook=cb)
    with pytest.raises(RuntimeError):
        ops.chain_rows(x, p, bits, n, k, codebook=cb[:-1])


@pytest.mark.parametrize("m,n,k,dtype,takes", [(64, 3072, 1024, torch.float32, True), (32, 6144, 2048, torch.bfloat16, True), (32, 2560, 2560, torch.float32, True),
                                               (64, 2560, 2560, torch.bfloat16, True), (40, 2560, 2560, torch.float32, False),
                                               (48, 6144, 2048, torch.bfloat16, False), (24, 7680, 2560, torch.float32, False), (65, 256, 256, torch.float32, False)])
def test_rows_that_are_faster_here_come_here(built_lib, m, n, k, dtype, takes):
    """The line between this kernel and the tcgen05 one, and that a call of PackedLinear on either side of it is right."""
    assert ops.chain_takes(m, n, k, 3, dtype) == takes
    packed, cb, _ = o.make_packed_linear(n, k, 3, seed=m)
    lin = PackedLinear(torch.from_numpy(packed).to(DEV), torch.from_numpy(cb).to(DEV), n, k)
    x = torch.randn(m, k, device=DEV, generator=torch.Generator(device=DEV).manual_seed(k)).to(dtype)
    want = x.double() @ lin.dequantized_weight().double().T
    for _ in range(2):                                     # the general path, then the native call
        _close(lin(x), want, {torch.float32: 10 * REL, torch.bfloat16: 2.0 ** -8}[dtype])       # (the GEMM's tolerance elsewhere is 2e-5 of max |y|)


def test_the_wrappers_refuse_what_does_not_fit(built_lib):
    """Sizes and types of every tensor are checked before a launch."""
    n, k, m, bits = 256, 128, 2, 3
    w, _ = _matrix(n, k, bits, 1)
    packed, cb, _ = o.make_packed_linear(n, k, bits, seed=1)
    packed, cb = torch.from_numpy(packed).to(DEV), torch.from_numpy(cb).to(DEV)
    f32 = dict(device=DEV, dtype=torch.float32)
    status, x, y = torch.zeros(1, dtype=torch.int32, device=DEV), torch.randn(m, k, **f32), torch.empty(m, n, **f32)
    sq, terms = torch.ones(m, k // 16, **f32), _terms(x)

    def linear(w=w, x_terms=terms, status=status, **kw):
        ops.chain_linear(ops.CHAIN_STORE, w, bits, m, n, k, x_terms, status, **{"y": y, **kw})
    linear()
    linear(x_terms=None, x=x, sq=sq, x_weight=torch.ones(k, **f32))
    linear(w=packed, codebook=cb)
    for bad in (dict(w=w[:-16]), dict(w=w.view(torch.int8)), dict(x_terms=terms[:-2]), dict(x_terms=terms.view(torch.float16)), dict(status=status.long()),
                dict(x_terms=None), dict(x=x), dict(x_terms=None, x=x[:, :-1]), dict(x_terms=None, x=x.half()), dict(sq=sq[0, :3]),
                dict(x_terms=None, x=x, sq=sq), dict(x_terms=None, x=x, sq=sq, x_weight=torch.ones(k - 1, **f32)), dict(w=packed[:-1], codebook=cb),
                dict(w=packed, codebook=cb[1:]), dict(w=packed, codebook=cb.double()), dict(y=y[:1]), dict(y=y.half()), dict(ahead=w.view(torch.int32)),
                dict(w=w.cpu()), dict(y_terms=terms.cpu())):
        with pytest.raises(RuntimeError):
            linear(**bad)
    for bad in ((w[:-16], None), (packed, cb[1:]), (packed[:-1], cb), (w.view(torch.int8), None)):
        with pytest.raises(RuntimeError):
            ops.chain_rows(x, bad[0], bits, n, k, codebook=bad[1])

    table, token = torch.randn(9, k, device=DEV).bfloat16(), torch.zeros(m, 1, dtype=torch.long, device=DEV)
    good = dict(table=table, token=token, weight=torch.ones(k, **f32), x=x, terms=terms, sq=sq)
    ops.chain_embed(**good)
    ops.chain_embed(**{**good, "weight": None, "terms": None})
    for bad in (dict(weight=torch.ones(k, device=DEV).half()), dict(weight=torch.ones(k - 1, **f32)), dict(table=table.float()), dict(table=table[:, 1:].contiguous()),
                dict(token=token.int()), dict(terms=terms[:-2]), dict(terms=terms.view(torch.float16)), dict(sq=sq[:1]), dict(x=x.half()), dict(sq=sq.half())):
        with pytest.raises(RuntimeError):
            ops.chain_embed(**{**good, **bad})

    heads, hd, ctx = 2, 64, 8
    good = dict(qkv=torch.randn(m, 3 * heads * hd, **f32), cos2=torch.ones(ctx, hd, **f32), sin2=torch.zeros(ctx, hd, **f32),
                pos=torch.zeros(1, dtype=torch.long, device=DEV), k_cache=torch.zeros(m, heads, ctx, hd, **f32), v_cache=torch.zeros(m, heads, ctx, hd, **f32),
                terms=ops.chain_terms(m, heads * hd, DEV), out_cols=heads * hd, out_offset=0)
    ops.decode_attention_terms(**good)
    for name, bad in (("qkv", good["qkv"][:, 1:].contiguous()), ("qkv", good["qkv"].half()), ("cos2", good["cos2"][:-1]), ("sin2", good["sin2"].double()),
                      ("pos", good["pos"].int()), ("k_cache", good["k_cache"].half()), ("v_cache", good["v_cache"][:, :, :-1].contiguous()),
                      ("k_cache", good["k_cache"].transpose(1, 2)), ("terms", good["terms"][:-2]), ("terms", good["terms"].view(torch.float16)),
                      ("qkv", good["qkv"].cpu())):
        with pytest.raises(RuntimeError):
            ops.decode_attention_terms(**{**good, name: bad})
    torch.cuda.synchronize()
