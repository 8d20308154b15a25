"""The stream-layout copies of PackedLinear's weights: complete before anybody finds them, made again together, never made by a
graph for others.  The packing itself is stubbed: it runs on a GPU only."""
import pytest
import torch

from nativebit_b200 import PackedLinear, packed_linear, stream
from nativebit_b200.packed_linear import make_copies


@pytest.fixture
def packing(monkeypatch):
    """Packs by copying, and notes the order of packings and waits."""
    log = []

    def pack(p, c, bits, n, k, row_mode=0, apart=True):
        log.append(("pack", row_mode))
        return torch.cat((p, c.view(torch.uint8).reshape(-1), torch.tensor([row_mode], dtype=torch.uint8)))
    monkeypatch.setattr(stream, "stream_pack", pack)
    monkeypatch.setattr(packed_linear, "_finish", lambda device, everything: log.append(("wait", everything)))
    return log


def _linear(seed):
    g = torch.Generator().manual_seed(seed)
    return PackedLinear(torch.randint(0, 256, (16 * 48,), dtype=torch.uint8, generator=g), torch.randn(16, 8, generator=g).half(), 16, 128)


def _is_of(w, lin, row_mode):
    return torch.equal(w, torch.cat((lin.packed_indices, lin.codebook.view(torch.uint8).reshape(-1), torch.tensor([row_mode], dtype=torch.uint8))))


def test_a_copy_is_complete_before_it_can_be_found(packing, monkeypatch):
    lin, other = _linear(0), _linear(1)
    found = []
    monkeypatch.setattr(packed_linear, "_finish", lambda device, everything: found.append(lin._copied_now() or other._copied_now()))
    make_copies([(lin, 0), (other, 0), (lin, 1)])
    assert packing == [("pack", 0), ("pack", 0), ("pack", 1)] and found and not any(found)
    assert lin._copied_now() and other._copied_now()
    make_copies([(lin, 0), (lin, 1), (other, 0)])
    assert len(packing) == 3


def test_both_copies_follow_other_weights_at_their_place(packing):
    lin, second = _linear(0), _linear(1)
    plain, gated = lin.stream_weight(0), lin.stream_weight(1)
    places = plain.data_ptr(), gated.data_ptr()
    lin.load_state_dict(second.state_dict())
    del packing[:]
    assert lin.stream_weight(0) is plain
    assert _is_of(plain, second, 0) and _is_of(gated, second, 1)              # the other one was not asked for
    assert packing[:3] == [("pack", 0), ("pack", 1), ("wait", True)]          # nothing launched over them is still running
    lin.codebook = _linear(2).codebook
    assert lin.stream_weight(1) is gated and _is_of(plain, lin, 0) and _is_of(gated, lin, 1)
    assert places == (plain.data_ptr(), gated.data_ptr())


@pytest.mark.parametrize("first", [True, False])
def test_copies_are_made_again_inside_and_outside_of_inference_mode(packing, first):
    """A copy that was made under inference mode is an inference tensor, which nothing outside of it may write to."""
    lin, second = _linear(0), _linear(1)
    with torch.inference_mode(first):
        w = lin.stream_weight()
    lin.load_state_dict(second.state_dict())
    with torch.inference_mode(not first):
        assert lin.stream_weight() is w and _is_of(w, second, 0)
        lin.packed_indices.add_(1)
        assert _is_of(lin.stream_weight(), lin, 0)


def test_a_graph_that_is_captured_makes_no_copy_for_others(packing, monkeypatch):
    lin = _linear(0)
    monkeypatch.setattr(packed_linear, "capturing", lambda device: True)
    assert lin._copy() is None
    own = lin.stream_weight()
    assert _is_of(own, lin, 0) and not lin._copied_now() and lin.stream_weight() is not own
    assert not any(what == "wait" for what, _ in packing)
    monkeypatch.setattr(packed_linear, "capturing", lambda device: False)
    w = lin.stream_weight()
    monkeypatch.setattr(packed_linear, "capturing", lambda device: True)
    assert lin._copy() is w


def test_native_check_of_many_copies(packing, built_lib):
    from nativebit_b200 import _lib
    lins = [_linear(i) for i in range(3)]
    make_copies([(lin, 0) for lin in lins])
    held = [(lin._buffers, lin._wstream_of) for lin in lins]
    assert _lib.bind().all_current(held) and _lib.bind().all_current([])
    lins[1].packed_indices.add_(1)
    assert not _lib.bind().all_current(held)
    make_copies([(lin, 0) for lin in lins])
    assert not _lib.bind().all_current(held)                                  # as of the old ones
    held = [(lin._buffers, lin._wstream_of) for lin in lins]
    assert _lib.bind().all_current(held)
    lins[2].codebook = lins[2].codebook.clone()
    assert not _lib.bind().all_current(held)
    for wrong in ([1], [(1, 2)], [({}, ())], [({}, held[0][1])]):
        assert not _lib.bind().all_current(wrong)
    with pytest.raises(TypeError):
        _lib.bind().all_current(None)


def test_the_first_launch_over_other_weights_is_ordered():
    """Behind a load of other weights a launch over the packed bytes may not start beside the launch that writes them."""
    lin, other = _linear(0), _linear(1)
    assert lin._unseen() and not lin._unseen()
    lin.load_state_dict(other.state_dict())
    assert lin._unseen() and not lin._unseen()
    lin.codebook = other.codebook
    assert lin._unseen() and not lin._unseen()
