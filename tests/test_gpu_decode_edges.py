"""Block decode at the edges of its tiles: images one block or texel around
the 32-, 64- and 128-block tile widths, row pitches and outputs at every
4-byte alignment, against the oracle bit for bit, with the bytes around the
image untouched."""
import numpy as np
import pytest
import torch

from oracle import binding as ob
from test_gpu_texture import _bc7_blocks
from vk_gltf_viewer_gb300 import abi

pytestmark = pytest.mark.gpu

FORMATS = [abi.BC1, abi.BC2, abi.BC3, abi.BC4, abi.BC5, abi.BC1_OPAQUE, abi.BC7, abi.BC6H_UF16, abi.BC6H_SF16]
SIZES = [(1, 1), (127, 4), (128, 33), (130, 31), (133, 3), (256, 9), (259, 66), (511, 17), (516, 35)]


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("size", SIZES)
def test_tile_edges_and_alignments(renderer, fmt, size):
    w, h = size
    rng = np.random.default_rng(100 * fmt + w + h)
    n = ((w + 3) // 4) * ((h + 3) // 4)
    hdr = fmt in (abi.BC6H_UF16, abi.BC6H_SF16)
    if fmt == abi.BC7:
        blocks = _bc7_blocks(rng, n)
    else:
        blocks = rng.integers(0, 256, size=n * (8 if fmt in (abi.BC1, abi.BC4, abi.BC1_OPAQUE) else 16), dtype=np.uint8)
    dev = torch.from_numpy(blocks).cuda()
    if hdr:
        exp = ob.decode_bc6h(blocks, w, h, fmt == abi.BC6H_SF16).view(np.float16).astype(np.float32)
    else:
        exp = ob.decode_bc(fmt, blocks, w, h)
    exp = np.ascontiguousarray(exp).reshape(-1).view(np.uint32)
    call = renderer.lib.vkgv_decode_bc6h if hdr else renderer.lib.vkgv_decode_bc
    for shift in range(4):  # the output at each 4-byte alignment
        out = torch.full((exp.size + 16,), 0x5A5A5A5A, dtype=torch.int32, device="cuda")
        at = out[4 + shift:]
        abi.check(call(renderer.ctx, fmt, dev.data_ptr(), w, h, at.data_ptr(),
                       torch.cuda.current_stream().cuda_stream), renderer.ctx)
        got = out.cpu().numpy().view(np.uint32)
        assert np.array_equal(got[4 + shift:4 + shift + exp.size], exp)
        assert (got[:4 + shift] == 0x5A5A5A5A).all() and (got[4 + shift + exp.size:] == 0x5A5A5A5A).all()
