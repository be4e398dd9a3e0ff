"""The rules that depend on sizes alone (csrc/dmm_choice.h), compiled by themselves: no GPU needed."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148

_SHIM = """
#include "dmm_choice.h"
extern "C" void wide(int nb, int units, long long rest, int sms, int can_split, int atomic, long long *out) {
    const dmm::WideSplit s = dmm::wide_split(nb, units, rest, sms, can_split != 0, atomic != 0);
    out[0] = s.parts;
    out[1] = s.share;
}
extern "C" int planes(long long M, int n, const long long *N, const long long *K, const int *silu, int sms) {
    dmm::HandoverSize size;
    for (int i = 0; i < n; ++i) size.add(N[i], K[i], sms, silu[i] != 0);
    return dmm::planes_in_front(M, size);
}
extern "C" int planes_tp(long long M, int mode, long long N, long long K, int silu, int sms) {
    dmm::HandoverSize size;
    size.add(N, K, sms, silu != 0);
    return dmm::planes_in_front_tp(M, mode, size);
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("choice")
    (d / "shim.cpp").write_text(_SHIM)
    so = str(d / "shim.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "decode_matmul_b200", "csrc"), "-o", so, str(d / "shim.cpp")], check=True)
    return ctypes.CDLL(so)


def _wide(rules, nb, units, rest, can_split=True, atomic=False):
    out = (ctypes.c_longlong * 2)()
    rules.wide(nb, units, ctypes.c_longlong(rest), SMS, int(can_split), int(atomic), out)
    return out[0], bool(out[1])


# (columns, units of 128 k, tiles), and the CTAs beyond which the measured time only rises: twice as many cost a tenth more or
# worse, all 148 up to twice the time
@pytest.mark.parametrize("nb,units,tiles,most", [(48, 256, 1, 32), (64, 256, 1, 32), (48, 64, 1, 16), (64, 224, 1, 32), (48, 64, 2, 32),
                                                 (64, 64, 2, 32), (48, 32, 4, 64), (64, 32, 4, 64), (48, 64, 8, 64),
                                                 (48, 16, 8, 64), (48, 8, 16, 16), (64, 8, 16, 16)])
def test_a_wide_tile_is_not_split_further_than_pays(rules, nb, units, tiles, most):
    assert _wide(rules, nb, units, tiles)[0] <= most


@pytest.mark.parametrize("nb", [16, 32, 48, 64, 80, 128])
def test_a_wide_split_stays_in_range(rules, nb):
    for units in (1, 2, 3, 9, 32, 86, 224, 1024):
        for tiles in (1, 2, 3, 16, 43, 74, 75, 112, 147):
            for atomic in (False, True):
                parts, share = _wide(rules, nb, units, tiles, atomic=atomic)
                assert tiles <= parts <= max(tiles, min(SMS, tiles * units))
                assert share == (parts > tiles and not atomic and 32 < nb <= 64 and nb * parts >= 150 * tiles)
            assert _wide(rules, nb, units, tiles, can_split=False) == (tiles, False)


def _planes(rules, M, *products):
    n = len(products)
    N, K = (ctypes.c_longlong * n)(*[p[0] for p in products]), (ctypes.c_longlong * n)(*[p[1] for p in products])
    return bool(rules.planes(ctypes.c_longlong(M), n, N, K, (ctypes.c_int * n)(*[p[2] for p in products]), SMS))


def _block(hidden, kv, ffn):
    return (hidden + 2 * kv, hidden, 0), (hidden, hidden, 0), (2 * ffn, hidden, 0), (hidden, ffn, 1)


# One product by itself behind silu(gate) * up: the loaders' exponential costs more than the planes kernel long before the line
# of plain products.  N = 64 * SMS, K = 128 * t: t tiles per SM.
@pytest.mark.parametrize("M,plain,silu", [(4, 290, 40), (5, 144, 16), (6, 77, 16), (7, 63, 16), (8, 58, 16)])
def test_planes_in_front_of_one_product(rules, M, plain, silu):
    for t, kind in ((plain, 0), (silu, 1)):
        assert not _planes(rules, M, (64 * SMS, 128 * t, kind))
        assert _planes(rules, M, (64 * SMS, 128 * (t + 1), kind))
        assert not _planes(rules, M, *[(64 * SMS, 128 * t, kind)] * 4)
        assert _planes(rules, M, *[(64 * SMS, 128 * (t + 1), kind)] * 4)


# The blocks of a stack keep one choice, the plain lines: one product of four is behind silu.
@pytest.mark.parametrize("M,shape,planes", [(4, (8192, 1024, 28672), False), (5, (4096, 4096, 11008), False), (5, (8192, 1024, 28672), True),
                                            (8, (4096, 4096, 11008), False), (8, (5120, 5120, 13824), True)])
def test_planes_in_front_of_a_block(rules, M, shape, planes):
    assert _planes(rules, M, *_block(*shape)) == planes


def test_planes_by_rows_alone(rules):
    for kind in (0, 1):
        assert not any(_planes(rules, M, (57344, 8192, kind)) for M in (1, 2, 3))
        assert all(_planes(rules, M, (16, 32, kind)) for M in (9, 16, 17, 32))


# The consumer of the slots form (mode 3) never has planes; its producer (2) follows the plain lines; products that add into every
# rank's buffer (0) have them from 4 rows on.
@pytest.mark.parametrize("M", range(1, 9))
def test_planes_in_front_of_tensor_parallel_products(rules, M):
    line = {4: 290, 5: 144, 6: 77, 7: 63, 8: 58}.get(M)

    def tp(mode, t, silu=0):
        return bool(rules.planes_tp(ctypes.c_longlong(M), mode, ctypes.c_longlong(64 * SMS), ctypes.c_longlong(128 * t), silu, SMS))

    for silu in (0, 1):
        assert not tp(3, 1, silu) and not tp(3, 400, silu)
        assert tp(0, 1, silu) == tp(0, 400, silu) == (M >= 4)
        assert not tp(2, line or 400, silu)
        assert line is None or tp(2, line + 1, silu)
