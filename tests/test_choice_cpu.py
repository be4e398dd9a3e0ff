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
