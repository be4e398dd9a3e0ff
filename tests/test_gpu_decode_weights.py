"""decode_weights at the sizes where its work items end.  Needs a B200."""
import numpy as np
import pytest
import torch

import decode_matmul_b200 as dmm
from oracle import dmm_oracle as o

pytestmark = pytest.mark.gpu


# one strip, one k-tile; k-tiles that do not fill an item of four; fewer and more items than warps on the chip
@pytest.mark.parametrize("N,K", [(16, 32), (16, 96), (32, 128), (48, 160), (272, 1056), (4096, 544), (20480, 608)])
@pytest.mark.parametrize("f16", [True, False])
def test_sizes_bit_exact(N, K, f16):
    rng = np.random.default_rng(N + K)
    codes = rng.integers(-32768, 32768, size=(N, K // 8)).astype(np.int16)
    cb64 = np.ascontiguousarray(o.build_codebook_abs())
    tiled = torch.from_numpy(np.ascontiguousarray(o.tile_pack(codes))).cuda()
    if f16:
        cb16 = o.cb64_to_cb16(cb64)
        got = dmm.decode_weights(tiled, torch.from_numpy(cb16).cuda()).cpu().numpy()
        assert np.array_equal(got.view(np.uint16), o.decode_weights_f16(codes, cb16).view(np.uint16))
    else:
        got = dmm.decode_weights(tiled, torch.from_numpy(cb64).cuda()).cpu().numpy()
        assert np.array_equal(got, o.decode_weights(codes, cb64))
    assert dmm.status() == 0


def test_large_table_bytes():
    """Table bytes up to the int8 range, which only this kernel and the integer family accept."""
    rng = np.random.default_rng(1)
    cb64 = (rng.integers(-31, 31, size=(256, 8)) * 4 + 2).astype(np.int8).view(np.int64).reshape(256)
    codes = np.arange(65536, dtype=np.uint16).view(np.int16).reshape(512, 128)
    tiled = torch.from_numpy(np.ascontiguousarray(o.tile_pack(codes))).cuda()
    cb16 = (cb64.view(np.int8).reshape(256, 8).astype(np.float16) / np.float16(4)).astype(np.float16)
    want = o.decode_weights(codes, cb64)
    got = dmm.decode_weights(tiled, torch.from_numpy(cb16).cuda()).cpu().numpy()
    assert np.array_equal(got, (want.astype(np.float32) / 4).astype(np.float16))
    assert dmm.status() == 0
