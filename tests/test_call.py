"""PackedLinear's native call against the general path: same results, same refusals."""
import pytest
import torch

from nativebit_b200 import PackedLinear, _lib, ops


def test_native_call_leaves_everything_else_to_the_general_path(built_lib):
    call = _lib.bind().linear
    x, p, c = torch.zeros(2, 128), torch.zeros(48, dtype=torch.uint8), torch.zeros(1, 8).half()
    assert call(x, p, c, None, None, 1, 128, 3, True, {}, {}) is None                  # not on a GPU
    assert call(x.int(), p, c, None, None, 1, 128, 3, True, {}, {}) is None
    assert call(torch.nn.Parameter(x), p, c, None, None, 1, 128, 3, True, {}, {}) is None
    assert call(None, p, c, None, None, 1, 128, 3, True, {}, {}) is None
    with pytest.raises(TypeError):
        call(x, p, c)
    with pytest.raises(TypeError):
        call(x, p, c, None, None, "n", 128, 3, True, {}, {})


def _general(lin, x):
    """The call without its native form."""
    flat = x.reshape(-1, lin.in_features).contiguous()
    if 2 <= flat.shape[0] <= 16:
        y = ops.chain_rows(flat, lin.stream_weight(), lin.bits, lin.out_features, lin.in_features, ordered=True)
        z = ops.gemv(flat, lin.packed_indices, lin.codebook, lin.bits, 128, lin.out_features, lin.in_features, ordered=True)
        # the sums of two kernels in fp32, rounded: two results to either side of a tie are an ulp apart
        assert (y.double() - z.double()).norm() <= {torch.float32: 2e-6, torch.float16: 2.0 ** -10, torch.bfloat16: 2.0 ** -7}[x.dtype] * z.double().norm()
    elif flat.shape[0] == 1:
        y = ops.gemv(flat, lin.packed_indices, lin.codebook, lin.bits, 128, lin.out_features, lin.in_features, ordered=True)
    else:
        y = lin._forward_many(flat)
    return y.reshape(*x.shape[:-1], lin.out_features)


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_native_call_equals_the_general_path(built_lib, bits, dtype):
    n, k = 272, 640
    g = torch.Generator(device="cuda").manual_seed(bits)
    idx = torch.randint(0, 1 << bits, (n * k,), dtype=torch.uint8, device="cuda", generator=g)
    lin = PackedLinear(ops.pack(idx, bits), torch.randn(n * k // 128, 1 << bits, device="cuda", generator=g).half(), n, k, bits=bits)
    big = torch.randn(700, 2 * k, device="cuda", generator=g).to(dtype)
    forms = [big[0, :k], big[:1, :k], big[:16, :k].contiguous(), big[:16, :k], big[:17, :k].contiguous(), big[:17, :k], big[:600, k:].contiguous(),
             big[:12, :k].reshape(3, 4, k), big[:40, :k].reshape(2, 20, k), big[:24, :k].view(4, 6, k).transpose(0, 1), big[:0, :k]]
    odd = torch.zeros(4 * k + 8, device="cuda", dtype=dtype)[1:4 * k + 1].view(4, k)                # not on a 16-byte boundary
    odd.copy_(big[:4, :k])
    assert torch.equal(lin(odd), ops.gemv(odd, lin.packed_indices, lin.codebook, bits, 128, n, k, ordered=True))
    for turn in range(2):                                   # the first calls make the workspaces and the stream-layout copy
        for x in forms:
            if x.shape[0] == 0:
                with pytest.raises(RuntimeError):           # no rows: refused as before
                    lin(x)
                continue
            y, want = lin(x), _general(lin, x)
            assert y.shape == want.shape and y.dtype == want.dtype and y.is_contiguous() and not y.requires_grad
            assert torch.equal(y, want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for x in (forms[1], forms[4]):
            assert torch.equal(lin(x), _general(lin, x))
        with torch.cuda.graph(graph := torch.cuda.CUDAGraph(), stream=side):
            y = lin(forms[2])
        graph.replay()
    side.synchronize()
    assert torch.equal(y, _general(lin, forms[2]))
    for wrong in (big[:4], big[:4, :k].double(), big[:4, :k].int()):
        with pytest.raises(RuntimeError):
            lin(wrong)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 4, 16, 20, 300])
def test_other_weights_are_what_the_next_call_multiplies(built_lib, rows):
    n, k = 144, 256
    g = torch.Generator(device="cuda").manual_seed(rows)

    def weights():
        idx = torch.randint(0, 8, (n * k,), dtype=torch.uint8, device="cuda", generator=g)
        return ops.pack(idx, 3), torch.randn(n * k // 128, 8, device="cuda", generator=g).half()

    first, second, third = weights(), weights(), weights()
    lin = PackedLinear(first[0].clone(), first[1].clone(), n, k)
    x = torch.randn(rows, k, device="cuda", generator=g)

    def check(w):
        for _ in range(3):
            assert torch.equal(lin(x), PackedLinear(*w, n, k)(x))

    lin.stream_weight()
    check(first)
    held = lin.stream_weight()
    lin.load_state_dict({"packed_indices": second[0], "codebook": second[1]})
    check(second)
    lin.codebook = third[1]
    check((second[0], third[1]))
    lin.packed_indices = third[0]
    check(third)
    assert lin.stream_weight().data_ptr() == held.data_ptr()            # what a captured graph reads


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 2, 16])
def test_few_rows_multiply_the_packed_bytes_themselves(built_lib, rows):
    """No copy that could be of other weights: writes that PyTorch does not count are followed as well, and nothing is kept."""
    n, k = 144, 256
    g = torch.Generator(device="cuda").manual_seed(rows)

    def weights():
        return ops.pack(torch.randint(0, 8, (n * k,), dtype=torch.uint8, device="cuda", generator=g), 3), torch.randn(n * k // 128, 8, device="cuda", generator=g).half()

    w = [weights() for _ in range(3)]
    x = torch.randn(rows, k, device="cuda", generator=g)
    want = [PackedLinear(*v, n, k)(x) for v in w]
    lin = PackedLinear(w[0][0].clone(), w[0][1].clone(), n, k)
    assert torch.equal(lin(x), want[0]) and torch.equal(lin(x), want[0])
    lin.packed_indices.data.copy_(w[1][0])
    lin.codebook.data.copy_(w[1][1])
    torch.cuda.synchronize()
    assert torch.equal(lin(x), want[1])
    with torch.inference_mode():
        lin = PackedLinear(w[0][0].clone(), w[0][1].clone(), n, k)
        assert lin.packed_indices.is_inference() and torch.equal(lin(x), want[0])
        lin.load_state_dict({"packed_indices": w[2][0], "codebook": w[2][1]})
        torch.cuda.synchronize()
        assert torch.equal(lin(x), want[2])
    assert not any("wstream" in name for name in lin.__dict__)
