"""Packed linear module and free functions with the reference's names and argument meaning.

Mirrors inference/triton_kernel.py (BS/NE/TILE_N :18-20, dequant_matvec :119-140,
dequant_matvec_3bit :186-196, pack_indices_to_3bit :199-220, PackedLinear :223-286) and
inference/cuda_kernel.py (dequant_matvec_3bit_cuda :133-136).  Differences, all deliberate:
every batch size runs a fused kernel (the reference re-materialises the whole weight for
M > 1), errors are raised instead of being swallowed into a second backend, launches go to
torch's current stream, and 2-bit (K=4) codebooks are accepted as well as 3-bit.
"""
from __future__ import annotations

import numpy as np
import torch
from torch.nn.modules import module as _module

from . import _lib, ops

BS = 128      # weights per codebook block
NE = 8        # codebook entries per block at 3 bits
TILE_N = 32   # kept for signature compatibility; the B200 kernels pick their own tiling
GEMV_MAX_M = 16
FUSED_MAX_ROWS = 1024   # up to this many activation rows the weights are dequantised inside the GEMM kernel


def pack_indices_to_3bit(indices_uint8: torch.Tensor) -> torch.Tensor:
    """uint8 indices (0..7) -> flat 3-bit packed bytes, on the GPU (inference/triton_kernel.py:199-220)."""
    return ops.pack(indices_uint8.contiguous().reshape(-1), 3)


def dequant_matvec_3bit(x, packed_indices, codebook, N, K, tile_n=TILE_N):
    """y (N,) fp32 = W @ x for one activation vector, 3-bit packed indices
    (inference/triton_kernel.py:186-196)."""
    # the caller may have produced packed_indices on this stream a moment ago (dequant_matvec packs per
    # call): the launch is fully stream-ordered
    y = ops.gemv(x.reshape(1, int(K)).contiguous(), packed_indices, codebook.contiguous(), 3, BS, int(N), int(K),
                 out_dtype=torch.float32, ordered=True)
    return y.reshape(int(N))


def dequant_matvec_3bit_cuda(x, packed, codebook, N, K):
    """Same contract as inference/cuda_kernel.py:133-136."""
    return dequant_matvec_3bit(x, packed.view(-1), codebook, N, K)


def dequant_matvec(x, indices, codebook, N, K, tile_n=TILE_N):
    """y (N,) fp32 = W @ x with unpacked uint8 indices of shape (num_blocks, BS)
    (inference/triton_kernel.py:119-140).  The indices are packed on the device first."""
    packed = ops.pack(indices.contiguous().reshape(-1), 3)
    return dequant_matvec_3bit(x, packed, codebook, N, K)


COPIES = ("_wstream", "_wstream_rm1")          # by row mode


def _version(t: torch.Tensor) -> int:
    return -1 if t.is_inference() else t._version


def capturing(device: torch.device) -> bool:
    if device.type != "cuda":
        return False
    with torch.cuda.device(device):
        return torch.cuda.is_current_stream_capturing()


def make_copies(wanted) -> None:
    """Makes the stream-layout copies (linear, row mode) that are missing or of other weights than the linear's present ones, and
    waits for them: whatever thread or stream finds a copy, it is complete.  Copies that are made again stay at their place, which
    captured graphs hold, after everything that was launched over them; both copies of a linear are made again together, so that
    no step meets one of old and one of new weights."""
    from .stream import stream_pack
    todo: dict = {}
    for lin, row_mode in wanted:
        have, now = lin.__dict__, lin._copied_now()
        for mode, name in enumerate(COPIES):
            if (mode == row_mode or have.get(name) is not None) and not (now and have.get(name) is not None):
                todo[id(lin), mode] = (lin, mode)
    made, of = [], {}
    for lin, mode in todo.values():
        p, c, *_ = of.setdefault(lin, lin.weights_now())
        made.append((lin, COPIES[mode], stream_pack(p, c, lin.bits, lin.out_features, lin.in_features, mode, apart=False)))
    for device in {w.device for _, _, w in made}:
        _finish(device, any(w.device == device and lin.__dict__.get(name) is not None for lin, name, w in made))
    again = set()
    for lin, name, w in made:
        old = lin.__dict__.get(name)
        if old is not None and old.device == w.device and old.shape == w.shape:
            with torch.inference_mode():        # either may be an inference tensor
                old.copy_(w)
            again.add(w.device)
        else:
            setattr(lin, name, w)
    for device in again:
        _finish(device, False)
    for lin, key in of.items():
        lin._wstream_of = key


def _finish(device: torch.device, everything: bool) -> None:
    """Waits for what the current stream, or the whole device, has been given."""
    if device.type == "cuda":
        torch.cuda.synchronize(device) if everything else torch.cuda.current_stream(device).synchronize()


class PackedLinear(torch.nn.Module):
    """Drop-in for nn.Linear over NativeBit packed weights (inference/triton_kernel.py:223-286).

    Buffers keep the reference's names: `packed_indices` (flat uint8 in the nativebit/pack.py
    layout) and `codebook` ((num_blocks, 2**bits), fp16 or fp32).  forward accepts any leading
    dims; the result has x's dtype.  Calls of up to 16 rows and of more than 1024 (512 of fp32) multiply these
    buffers; those between keep a tile-major copy of them (stream_weight), which the first such call makes and waits for.
    """

    def __init__(self, packed_indices, codebook, out_features, in_features, bits: int = 3, block_size: int = BS):
        super().__init__()
        self.register_buffer("packed_indices", packed_indices)
        self.register_buffer("codebook", codebook)
        self.out_features = int(out_features)
        self.in_features = int(in_features)
        self.bits = int(bits)
        self.block_size = int(block_size)
        # The buffers may have been written by kernels still in flight (from_packed / pack_linear pack on the device, weights are
        # loaded): the first launch over other weights than these is fully stream-ordered, later ones may start early.
        self._seen = []

    def forward(self, x):
        if self.block_size == BS and x.is_cuda:      # the plain calls: checks, result and launch in one native function
            y = _lib.bind().linear(x, self.packed_indices, self.codebook, self.__dict__.get("_wstream"), self.__dict__.get("_wstream_of"),
                                   self.out_features, self.in_features, self.bits, self._seen, ops._workspaces, ops._prefill_ws)
            if y is not None:
                return y
        shape = x.shape
        x_flat = x.reshape(-1, self.in_features)
        if not x_flat.is_contiguous():
            x_flat = x_flat.contiguous()
        m = x_flat.shape[0]
        if self.block_size != BS or self.bits not in (2, 3, 4):
            # shapes outside the fused kernels (small codebook blocks): gather kernel + matmul
            w = ops.dequant(self.packed_indices, self.codebook, self.bits, self.block_size,
                            (self.out_features, self.in_features),
                            dtype=x_flat.dtype if x_flat.dtype in (torch.float16, torch.bfloat16) else torch.float32)
            y = x_flat @ w.T
        elif 2 <= m <= GEMV_MAX_M and (y := self._forward_few(x_flat)) is not None:
            pass
        elif m <= GEMV_MAX_M:
            y = ops.gemv(x_flat, self.packed_indices, self.codebook, self.bits, self.block_size,
                         self.out_features, self.in_features, ordered=self._unseen())
        else:
            y = self._forward_many(x_flat)
        return y.reshape(*shape[:-1], self.out_features)

    def stream_weight(self, row_mode: int = 0):
        """Tile-major copy of the packed weight for the fused tensor-core kernel and the many-matrix / decode-chain
        kernels: made on first use, kept with the module at one place in memory, made again after other weights were loaded or
        assigned (not after writes that PyTorch does not count: through `.data`, or to inference tensors).  row_mode 1: this is a fused
        [gate | up] matrix and every 16-row tile holds 8 gate channels and the matching 8 up channels (for a SwiGLU epilogue)."""
        w = self._copy(row_mode)
        if w is None:                       # under capture: the graph's own copy, packed by every replay
            from .stream import stream_pack
            w = stream_pack(self.packed_indices, self.codebook, self.bits, self.out_features, self.in_features, row_mode)
        return w

    def _copy(self, row_mode: int = 0):
        """stream_weight, but None under capture where the copy would have to be made."""
        if not self._copied_now() or self.__dict__.get(COPIES[row_mode]) is None:
            if capturing(self.packed_indices.device):
                return None
            make_copies([(self, row_mode)])
        return self.__dict__[COPIES[row_mode]]

    def _unseen(self) -> bool:
        """Whether the launch that follows is the first over the packed bytes as they are now."""
        now, seen = self.weights_now(), self._seen
        if len(seen) == 4 and seen[0] is now[0] and seen[1] is now[1] and (seen[2], seen[3]) == now[2:]:
            return False
        seen[:] = now
        return True

    def weights_now(self) -> tuple:
        """The tensors and versions that a copy made now is of."""
        p, c = self.packed_indices, self.codebook
        return p, c, _version(p), _version(c)

    def _copied_now(self) -> bool:
        """Whether the copies are of the weights as they are now."""
        of = self.__dict__.get("_wstream_of")
        return of is not None and of[0] is self.packed_indices and of[1] is self.codebook and of[2:] == (_version(of[0]), _version(of[1]))

    def _forward_few(self, x_flat):
        """2 to 16 rows on the chain's kernel over the packed bytes, None where nb_gemv takes them."""
        if not ops.chain_takes_packed(x_flat.shape[0], self.out_features, self.in_features, self.bits, x_flat.dtype) or x_flat.data_ptr() % 16 or self.packed_indices.data_ptr() % 16 or self.codebook.data_ptr() % 16:
            return None
        y = ops.chain_rows(x_flat, self.packed_indices, self.bits, self.out_features, self.in_features, ordered=self._unseen(),
                           codebook=self.codebook)
        if y is None:
            self._seen.clear()              # nothing was launched
        return y

    def _forward_many(self, x_flat):
        """M > 16 rows on the tcgen05 kernels (exact fp16 weights; bf16 and fp16 activations as given, fp32
        carried as two fp16 terms; fp32 accumulation; result in x's dtype): one pass over the packed weights,
        dequantised inside the kernel, up to FUSED_MAX_ROWS rows; dequantise-once + GEMM beyond."""
        if (x_flat.dtype in (torch.float32, torch.float16, torch.bfloat16) and x_flat.data_ptr() % 16 == 0
                and self._few_enough(x_flat.shape[0], x_flat.dtype) and (w := self._copy()) is not None
                and (y := ops.chain_rows(x_flat, w, self.bits, self.out_features, self.in_features)) is not None):
            return y
        if self._tensor_cores():
            rows = x_flat.shape[0] * (2 if x_flat.dtype == torch.float32 else 1)
            if rows > FUSED_MAX_ROWS or (w := self._copy()) is None:
                # long inputs: dequantising W once into a scratch copy (8.8 us for 6912 x 2560) and running the plain
                # tensor-core kernel, against dequantising every weight tile once per 256 operand rows.  6912 x 2560, fused |
                # two passes (us): bf16 512 rows 30.0 | 31.8, 1024 45 | 42, 2048 71 | 67; fp32 512 rows 37 | 44, 1024 59 | 68, 2048
                # 117 | 118.  bf16 rows cross between 256 (2560 x 2560) and 1280 (13824 x 2560), fp32 ones only past 1024:
                # up to there the line is early for them by up to a seventh.
                return ops.gemm_prefill(x_flat, self.packed_indices, self.codebook, self.bits, self.block_size,
                                        self.out_features, self.in_features, out_dtype=x_flat.dtype)
            return ops.gemm_prefill_fused(x_flat, w, self.bits, self.out_features, self.in_features,
                                          out_dtype=x_flat.dtype)
        wdt = x_flat.dtype if x_flat.dtype in (torch.float16, torch.bfloat16) else torch.float32
        w = ops.dequant(self.packed_indices, self.codebook, self.bits, self.block_size,
                        (self.out_features, self.in_features), dtype=wdt)
        return x_flat @ w.T

    def _tensor_cores(self) -> bool:
        return self.block_size == BS and self.in_features % BS == 0 and self.bits in (2, 3, 4)

    def _few_enough(self, rows: int, dtype) -> bool:
        """More than 16 rows, of a matrix so small that they are faster on the kernel for few rows."""
        return self._tensor_cores() and ops.chain_takes(rows, self.out_features, self.in_features, self.bits, dtype)

    def takes_terms(self, rows: int) -> bool:
        """Whether a call would split this many fp32 rows into two fp16 terms itself and nobody else looks at them, so that
        `forward_terms` may take their place: no hooks, no forward of a subclass or of this instance."""
        seen = (self._forward_pre_hooks or self._forward_hooks or _module._global_forward_pre_hooks or _module._global_forward_hooks
                or "forward" in self.__dict__ or type(self).forward is not PackedLinear.forward)
        return rows > GEMV_MAX_M and self._tensor_cores() and not self._few_enough(rows, torch.float32) and not seen

    def forward_terms(self, terms, out=None):
        """fp32 (M, out_features) of M fp32 rows given as their two fp16 terms, (2M, in_features); see ops.add_rmsnorm_terms."""
        if not self._tensor_cores():
            raise RuntimeError(f"forward_terms needs 2 to 4 bits, blocks of {BS} and a multiple of {BS} columns: {self.extra_repr()}")
        if terms.shape[0] > FUSED_MAX_ROWS or (w := self._copy()) is None:
            return ops.gemm_prefill(terms, self.packed_indices, self.codebook, self.bits, self.block_size, self.out_features, self.in_features,
                                    out_dtype=torch.float32, out=out, terms=True)
        return ops.gemm_prefill_fused(terms, w, self.bits, self.out_features, self.in_features, out=out, terms=True)

    def dequantized_weight(self, dtype=torch.float32):
        """The dense (out_features, in_features) weight; bit-exact gather of the codebook values."""
        return ops.dequant(self.packed_indices, self.codebook, self.bits, self.block_size,
                           (self.out_features, self.in_features), dtype=dtype)

    @staticmethod
    def from_packed(indices_np, codebook_np, weight_shape, device="cuda", bits: int = 3):
        """From unpacked uint8 numpy indices + codebook as stored in .nbpack.npz
        (inference/triton_kernel.py:277-286): indices are packed on the GPU."""
        indices_uint8 = torch.from_numpy(np.ascontiguousarray(indices_np)).to(device)
        packed = ops.pack(indices_uint8.reshape(-1), bits)
        codebook = torch.from_numpy(np.ascontiguousarray(codebook_np)).to(device)
        return PackedLinear(packed, codebook, weight_shape[0], weight_shape[1], bits=bits)

    def extra_repr(self):
        return f"in_features={self.in_features}, out_features={self.out_features}, bits={self.bits}"
