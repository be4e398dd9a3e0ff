"""Which kernel DMM_PATH_AUTO takes, at both sides of each line of wide_is_faster.  The plane kernels and the wide one
add in another order, so their results differ in the last bits, and each gives the same bits every time: a call on
DMM_PATH_AUTO that equals DMM_PATH_TCGEN05_F8 bit for bit ran on the planes.  Needs a B200."""
import pytest
import torch

import decode_matmul_b200 as dmm
from decode_matmul_b200 import _lib, ops
from oracle import dmm_oracle as o

pytestmark = pytest.mark.gpu


def _on_planes(M, t, x_kind):
    """Whether a product of M rows with t tiles per SM runs on the plane kernels."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    N, K = 64 * sms, 128 * t  # sms / 4 super-tiles of 4 t k-tiles: 0.8 t tiles per segment
    assert sms % 4 == 0
    gen = torch.Generator(device="cuda").manual_seed(t)
    codes = torch.randint(-32768, 32768, (N, K // 8), dtype=torch.int16, device="cuda", generator=gen)
    cb = torch.from_numpy(o.synthetic_codebook(42)).cuda()
    ld = 2 * K if x_kind == _lib.X_F32_SILU_MUL else K
    x = torch.randn((M, ld), device="cuda", generator=gen).to(torch.float16 if x_kind == _lib.X_F16 else torch.float32)
    got = []
    for path in (_lib.PATH_AUTO, _lib.PATH_TCGEN05_F8):
        y = torch.empty((M, N), device="cuda")
        rc = _lib.lib().dmm_f16_fused(x.data_ptr(), x_kind, ld, K if ld > K else 0, codes.data_ptr(), cb.data_ptr(), 1.0,
                                      y.data_ptr(), M, N, K, _lib.SIGN_SLOW, _lib.LAYOUT_TILE, path, 0, None, 0, None, 0,
                                      ops._stream_ptr(x.device))
        assert rc == 0
        got.append(y)
    # Both are within 1e-6 of the exact product.  Behind silu with the fast exponential an activation may round to the
    # other half here and there (2^-11 of it): 1e-4, as where the wide kernel is compared with the oracle.
    assert float((got[0] - got[1]).norm() / got[1].norm()) <= (1e-4 if x_kind == _lib.X_F32_SILU_MUL else 2e-6)
    assert dmm.status() == 0
    return torch.equal(got[0], got[1])


@pytest.mark.parametrize("M,x_kind,limit", [
    (4, _lib.X_F16, 32), (6, _lib.X_F16, 49), (8, _lib.X_F16, 59), (9, _lib.X_F16, 90), (12, _lib.X_F16, 123), (16, _lib.X_F16, 167),
    (9, _lib.X_F32, 49), (16, _lib.X_F32, 56), (16, _lib.X_F32_SILU_MUL, 56), (17, _lib.X_F32, 62), (32, _lib.X_F32, 62),
    (17, _lib.X_F32_SILU_MUL, 107), (32, _lib.X_F32_SILU_MUL, 107)])
def test_lines(M, x_kind, limit):
    assert not _on_planes(M, limit, x_kind)
    assert _on_planes(M, limit + 1, x_kind)


@pytest.mark.parametrize("M,x_kind,t,planes", [(3, _lib.X_F16, 1, True), (8, _lib.X_F32, 1, True), (17, _lib.X_F16, 220, False),
                                               (33, _lib.X_F32, 220, False)])
def test_beyond_the_lines(M, x_kind, t, planes):
    assert _on_planes(M, t, x_kind) == planes


# batch 1 and 2: two k-tiles per hand-over where segments are short, four on the others (HandoverSize: 28 tiles per
# segment; with 148 SMs the line lies between 2496 and 2528 at 82 super-tiles); numbers of k-tiles that neither divides
@pytest.mark.parametrize("N,K", [(16, 32), (272, 2048), (20992, 2496), (20992, 2528), (20976, 2656), (57344, 1056), (57344, 1600),
                                 (4112, 8256), (4112, 10528)])
@pytest.mark.parametrize("M", [1, 2])
def test_hand_over_of_two_and_of_four(M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    codes = torch.randint(-32768, 32768, (N, K // 8), dtype=torch.int16, device="cuda", generator=gen)
    cb = torch.from_numpy(o.synthetic_codebook(42)).cuda()
    x = torch.randn((M, K), device="cuda", generator=gen).to(torch.float16)
    w = dmm.decode_weights(codes, cb)
    want = torch.cat([x.double() @ part.double().T for part in w.split(16384)], dim=1)
    base = torch.randn((M, N), device="cuda", generator=gen)
    # exact products, sums off by the truncation of the tensor core: 7e-7 to 9e-7 at any length
    for out, kw, ref in ((None, {}, want), (base.clone(), dict(accumulate=True, atomic=True), want + base)):
        y = dmm.decode_matmul_fp16(x, codes, cb, 1.0, out, **kw).double()
        assert float((y - ref).norm() / ref.norm()) <= 2e-6
    assert dmm.status() == 0
