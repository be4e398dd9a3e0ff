"""The wide fp16-operand kernel (larger batches, and smaller ones on small matrices) against the CPU oracle, at the sizes where its tiles,
units and splits end.  Needs a B200."""
import numpy as np
import pytest
import torch

import decode_matmul_b200 as dmm
from decode_matmul_b200 import _lib
from oracle import dmm_oracle as o

pytestmark = pytest.mark.gpu

# Products of a half and an odd multiple of 1/4 are exact in fp32, so the only error is that of the fp32 sums: with
# K terms each addition is off by at most 2^-23 of the running sum (tensor cores may truncate), and the running
# sums of random terms stay within a few times the result's root mean square.  K <= 2048 terms in steps of 16
# are 128 additions; their errors add like a random walk with drift: 128 * 2^-23 = 1.5e-5 at the very worst.
REL = 1.5e-5


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    assert dmm.status() == 0, "a kernel raised the device status word"


def _case(M, N, K, seed=0, codebook="e8p"):
    rng = np.random.default_rng(M * 1000003 + N * 101 + K + seed)
    x = rng.standard_normal((M, K)).astype(np.float16)
    codes = rng.integers(-32768, 32768, size=(N, K // 8)).astype(np.int16)
    cb16 = o.cb64_to_cb16(np.ascontiguousarray(o.build_codebook_abs())) if codebook == "e8p" else o.synthetic_codebook(42)
    return x, codes, cb16


def _want(x, codes, cb16, convention=None):
    w = o.decode_weights_f16(codes, cb16) if convention is None else o.decode_weights_f16(codes, cb16, convention)
    return x.astype(np.float64) @ w.astype(np.float64).T


def _rel(y, want):
    return np.linalg.norm(y.astype(np.float64) - want) / np.linalg.norm(want)


# rows around every column-tile size (64, 128, 192 and their multiples), N around 256, K around 64 and 128
SHAPES = [(4, 16, 32), (5, 528, 1056), (16, 512, 160), (17, 16, 32), (17, 272, 64), (31, 256, 96), (32, 528, 1056), (33, 240, 2048), (48, 4096, 544), (64, 512, 512),
          (65, 512, 160), (128, 272, 1024), (129, 256, 2048), (192, 320, 128), (193, 528, 1056), (333, 1024, 512),
          (400, 16, 96), (577, 4096, 128), (1000, 9472, 64)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_shapes(M, N, K):
    x, codes, cb16 = _case(M, N, K, codebook="e8p" if M % 2 else "synthetic")
    want = _want(x, codes, cb16)
    tiled, cb = _dev(o.tile_pack(codes)), _dev(cb16)
    first = None
    for _ in range(2):  # the second call checks that the workspace counters were reset
        y = dmm.decode_matmul_fp16(_dev(x), tiled, cb).cpu().numpy()
        assert _rel(y, want) <= REL
        assert first is None or np.array_equal(first, y), "the summation order must be fixed"
        first = y


@pytest.mark.parametrize("M", [24, 100, 200])
def test_fast_layout_and_convention(M):
    x, codes, cb16 = _case(M, 544, 1056, 1)
    want = _want(x, codes, cb16, o.SIGN_FAST)
    y = dmm.decode_matmul_fp16(_dev(x), dmm.fast_pack(_dev(codes)), _dev(cb16), sign_convention=_lib.SIGN_FAST,
                               layout=_lib.LAYOUT_FAST).cpu().numpy()
    assert _rel(y, want) <= REL


@pytest.mark.parametrize("M", [20, 70, 333])
@pytest.mark.parametrize("atomic", [False, True])
def test_accumulate_and_scale(M, atomic):
    x, codes, cb16 = _case(M, 768, 1024, 2)
    base = np.random.default_rng(3).standard_normal((M, 768)).astype(np.float32)
    out = _dev(base)
    y = dmm.decode_matmul_fp16(_dev(x), _dev(o.tile_pack(codes)), _dev(cb16), 0.125, out, accumulate=True, atomic=atomic)
    assert y.data_ptr() == out.data_ptr()
    assert _rel(y.cpu().numpy(), base + 0.125 * _want(x, codes, cb16)) <= REL


@pytest.mark.parametrize("M", [9, 16, 17, 64, 65, 150])
@pytest.mark.parametrize("silu", [False, True])
def test_fp32_inputs_and_clearing(M, silu):
    """fp32 activations are rounded to fp16 first, as the narrower kernels do; `zero` is cleared on the way."""
    N, K = 288, 1056
    x, codes, cb16 = _case(M, N, K, 4)
    rng = np.random.default_rng(5)
    xf = rng.standard_normal((M, 2 * K if silu else K)).astype(np.float32)
    xt = torch.from_numpy(xf)
    half = (torch.nn.functional.silu(xt[:, :K]) * xt[:, K:] if silu else xt).to(torch.float16).numpy()
    zero = torch.full((1000,), 7.0, device="cuda")
    out = torch.zeros((M, N), device="cuda")
    dmm.decode_matmul_fused(_dev(xf), _dev(o.tile_pack(codes)), _dev(cb16), 1.0, out,
                            x_kind=_lib.X_F32_SILU_MUL if silu else _lib.X_F32, x_gap=K if silu else 0, accumulate=True,
                            atomic=True, zero=zero)
    # silu in the kernel uses the fast exponential: its rounding to half can differ by an ulp here and there
    assert _rel(out.cpu().numpy(), _want(half, codes, cb16)) <= (1e-4 if silu else REL)
    assert float(zero.abs().max()) == 0.0


@pytest.mark.parametrize("M", [4, 9, 16, 17, 33, 70, 200])
@pytest.mark.parametrize("layout", ["tile", "fast"])
@pytest.mark.parametrize("convention", ["slow", "fast"])
def test_same_as_the_plane_kernels(M, layout, convention):
    """The path that the library picks against the fp8-plane kernels, over layouts, sign conventions and results that
    are written or added.  Each is within 1e-6 of the exact product (the planes 8e-7, the halves 6.2e-7)."""
    N, K = 800, 672
    x, codes, cb16 = _case(M, N, K, 9, "synthetic")
    codes = _dev(codes)
    packed = dmm.fast_pack(codes) if layout == "fast" else dmm.transpose_tile(codes)
    kw = dict(layout=_lib.LAYOUT_FAST if layout == "fast" else _lib.LAYOUT_TILE,
              sign_convention=_lib.SIGN_FAST if convention == "fast" else _lib.SIGN_SLOW)
    base = torch.randn((M, N), device="cuda")
    for accumulate, atomic in ((False, False), (True, False), (True, True)):
        got = []
        for path in (_lib.PATH_AUTO, _lib.PATH_TCGEN05_F8):
            out = base.clone()
            dmm.decode_matmul_fp16(_dev(x), packed, _dev(cb16), 0.5, out, path=path, accumulate=accumulate, atomic=atomic, **kw)
            got.append(out.cpu().numpy())
        assert _rel(got[0], got[1].astype(np.float64)) <= 2e-6


def test_wide_rows_of_a_larger_buffer():
    """Rows of x that lie further apart than K (fp16 and fp32), as a layer reads a part of the one before."""
    M, N, K, ld = 40, 288, 544, 800
    x, codes, cb16 = _case(M, N, ld, 10)
    codes = np.ascontiguousarray(codes[:, : K // 8])
    want = _want(np.ascontiguousarray(x[:, :K]), codes, cb16)
    tiled, cb = _dev(o.tile_pack(codes)), _dev(cb16)
    for t, kind in ((_dev(x), _lib.X_F16), (_dev(x.astype(np.float32)), _lib.X_F32)):
        out = torch.empty((M, N), device="cuda")
        dmm.decode_matmul_fused(t, tiled, cb, 1.0, out, x_kind=kind)
        assert _rel(out.cpu().numpy(), want) <= REL


def _device_case(M, N, K, x_positive=False, w_positive=False):
    """Inputs made on the GPU, for sizes that are too large for the oracle: x, tiled codes, table, and the product in 64 bits
    from decode_weights, which equals the oracle's decode bit for bit (test_gpu_decode_weights.py)."""
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    cb = _dev(o.cb64_to_cb16(np.ascontiguousarray(o.build_codebook_abs())))
    if w_positive:
        table = o.decode_table(np.ascontiguousarray(o.build_codebook_abs()), o.SIGN_SLOW).reshape(65536, 8)
        words = _dev(np.arange(65536, dtype=np.uint16).view(np.int16)[(table > 0).all(1)])
        codes = words[torch.randint(0, len(words), (N, K // 8), device="cuda", generator=gen)]
    else:
        codes = torch.randint(-32768, 32768, (N, K // 8), dtype=torch.int16, device="cuda", generator=gen)
    x = torch.randn((M, K), device="cuda", generator=gen).to(torch.float16)
    x = x.abs() if x_positive else x
    want = torch.empty((M, N), dtype=torch.float64, device="cuda")
    for n0 in range(0, N, 8192):
        rows = dmm.decode_weights(dmm.transpose_tile(codes[n0:n0 + 8192]), cb).double()
        want[:, n0:n0 + 8192] = x.double() @ rows.T
    return x, dmm.transpose_tile(codes), cb, want


def _off(y, want):
    return float((y.double() - want).norm() / want.norm())


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


# One tile more than there are CTAs and one less than half as many again: every CTA has a whole tile of 25 units (three
# chains in each build: 32, 64 and 128 columns, the last one also as three column tiles of 112), and some a part of a split
# one behind it, which ends with a quarter of a unit.  The rows end in the last strip but one of a super-tile.
@pytest.mark.parametrize("rest", [1, 68])
@pytest.mark.parametrize("M", [20, 64, 128, 333])
def test_whole_tiles_of_several_chains_and_split_ones(M, rest):
    K = 3104
    N = 256 * ((_sms() + rest + 2) // (3 if M == 333 else 1)) - 16
    x, tiled, cb, want = _device_case(M, N, K)
    base = torch.randn((M, N), device="cuda")
    first = dmm.decode_matmul_fp16(x, tiled, cb)
    assert _off(first, want) <= 1e-6  # see test_error_of_long_reductions
    assert torch.equal(first, dmm.decode_matmul_fp16(x, tiled, cb)), "the summation order must be fixed"
    for atomic in (False, True):
        y = dmm.decode_matmul_fp16(x, tiled, cb, 1.0, base.clone(), accumulate=True, atomic=atomic)
        assert _off(y, want + base) <= 1e-6


# The tensor core truncates when it adds to its accumulator.  Cut into chains of at most 88 MMAs the sums of random terms
# were off by at most 6.2e-7, whatever the length; not cut, by 2.6e-5 at this one.  Terms of one sign are the
# worst case, since the truncations then add up: each takes at most 2^-23 of a sum that grows evenly, so at most
# 88 * 2^-23 / 2 = 5.2e-6 over a chain and about a quarter of that for uniform mantissas and remainders; measured 1.3e-6.
@pytest.mark.parametrize("one_signed", [False, True])
@pytest.mark.parametrize("M,tiles", [(16, 1), (17, 148), (64, 1), (64, 148), (100, 148), (128, 148), (333, 50)])
def test_error_of_long_reductions(M, tiles, one_signed):
    x, tiled, cb, want = _device_case(M, 256 * tiles, 28672, one_signed, one_signed)
    assert _off(dmm.decode_matmul_fp16(x, tiled, cb), want) <= (2e-6 if one_signed else 1e-6)


def test_small_workspace_leaves_the_tiles_whole():
    """A caller's workspace that only fits the narrower kernels is accepted and not written past its end; the tiles that are
    split in one of the full size (whose sums then come out in another order) are computed whole."""
    M, N, K = 128, 256 * (_sms() + 68) - 16, 3104
    x, tiled, cb, want = _device_case(M, N, K)
    full = dmm.workspace_bytes(M, N, K)
    small = dmm.workspace_bytes(64, N, K)
    assert small < full - 256
    got = []
    for size in (full, full - 256, small):
        room = torch.zeros((full + (64 << 20),), dtype=torch.uint8, device="cuda")
        room[size:] = 0x5A
        out = torch.empty((M, N), device="cuda")
        dmm.decode_matmul_fused(x, tiled, cb, 1.0, out, x_kind=_lib.X_F16, workspace=room[:size])
        assert _off(out, want) <= 1e-6
        assert bool((room[size:] == 0x5A).all())
        got.append(out)
    assert torch.equal(got[1], got[2]) and not torch.equal(got[0], got[1])


# the kernel's own loaders (up to 16 rows) and half_kernel in front of it, over the layout of fast_decode_matmul_cuda, which only
# the C entry combines with fp32 activations
@pytest.mark.parametrize("M", [9, 16, 24])
@pytest.mark.parametrize("silu", [False, True])
def test_fast_layout_with_fp32_inputs(M, silu):
    N, K = 544, 1056
    x, codes, cb16 = _case(M, N, K, 11)
    rng = np.random.default_rng(12)
    xf = rng.standard_normal((M, 2 * K if silu else K)).astype(np.float32)
    xt = torch.from_numpy(xf)
    half = (torch.nn.functional.silu(xt[:, :K]) * xt[:, K:] if silu else xt).to(torch.float16).numpy()
    want = _want(half, codes, cb16, o.SIGN_FAST)
    xd, packed, cb = _dev(xf), dmm.fast_pack(_dev(codes)), _dev(cb16)
    base = np.random.default_rng(13).standard_normal((M, N)).astype(np.float32)
    for flags in (0, _lib.FLAG_ACCUMULATE | _lib.FLAG_ATOMIC):
        out = _dev(base)
        rc = _lib.lib().dmm_f16_fused(xd.data_ptr(), _lib.X_F32_SILU_MUL if silu else _lib.X_F32, xd.shape[1], K if silu else 0,
                                      packed.data_ptr(), cb.data_ptr(), 1.0, out.data_ptr(), M, N, K, _lib.SIGN_FAST,
                                      _lib.LAYOUT_FAST, _lib.PATH_AUTO, flags, None, 0, None, 0,
                                      torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        # (silu uses the fast exponential, see test_fp32_inputs_and_clearing)
        assert _rel(out.cpu().numpy(), want + (base if flags else 0)) <= (1e-4 if silu else REL)


@pytest.mark.parametrize("batch", [9, 16, 24])
def test_fused_step_that_mixes_the_kernels(batch):
    """A block wide enough for the planes: of its four products one (o, at 24 rows also down) or none runs on the wide kernel.
    Same result as the step with separate conversions."""
    from decode_matmul_b200.linear import LinearStack

    cfg = dict(hidden=8192, kv_heads=8, head_dim=128, ffn=14336, layers=1)
    stack = LinearStack(cfg, dmm.synthetic_codebook(42), "cuda", seed=6, scale=2.0 ** -10)
    h0 = torch.randn(batch, 8192, device="cuda", generator=torch.Generator(device="cuda").manual_seed(batch))
    h_fused = stack.step(h0.clone(), fused=True)
    h_plain = stack.step(h0.clone(), fused=False, path=_lib.PATH_TCGEN05_F8)
    # Of what the block adds.  Both steps round the same intermediate sums to halves; one that falls to the other side is
    # off by 2^-11, and fewer than one in a hundred does: 2^-11 / 10.
    assert float((h_fused - h_plain).norm() / (h_plain - h0).norm()) <= 5e-5


@pytest.mark.parametrize("M", [32, 192])
def test_extreme_activations(M):
    """Largest and smallest halves: the weights are 2^-17 units inside the kernel, the result must not show it."""
    x, codes, cb16 = _case(M, 256, 256, 7)
    rng = np.random.default_rng(8)
    x[:, :] = rng.choice(np.array([65504, -65504, 6e-8, -6e-8, 0.0, 1.0], dtype=np.float16), size=x.shape)
    x[3, :] = np.float16(6e-8)
    want = _want(x, codes, cb16)
    y = dmm.decode_matmul_fp16(_dev(x), _dev(o.tile_pack(codes)), _dev(cb16)).cpu().numpy()
    assert _rel(y, want) <= REL
    assert _rel(y[3], want[3]) <= REL
    x[5, 7] = np.float16("inf")
    x[6, 9] = np.float16("nan")
    y = dmm.decode_matmul_fp16(_dev(x), _dev(o.tile_pack(codes)), _dev(cb16)).cpu().numpy()
    assert np.all(~np.isfinite(y[5])) and np.all(np.isnan(y[6])) and np.all(np.isfinite(np.delete(y, [5, 6], axis=0)))
