"""What a launch may read before the one in front of it has ended: weights that were written a moment ago, by another stream, or
under capture."""
import pytest
import torch

from nativebit_b200 import ops

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
