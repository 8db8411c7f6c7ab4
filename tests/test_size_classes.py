"""Launch size classes of the autotuner and the nearest usable choice (csrc/size_class.cuh, compiled
for the host)."""
import ctypes as ct
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "casadi_gb300",
                    "csrc")
SHIM = r"""
#include "size_class.cuh"
extern "C" {
int classes() { return cgb::kSizeClasses; }
int cls(long long items, int few, int sms) { return cgb::size_class(items, few != 0, sms); }
int kept(const int* row, int c, unsigned usable) {
  int r[cgb::kSizeClasses];
  for (int k = 0; k < cgb::kSizeClasses; ++k) r[k] = row[k];
  return cgb::kept_choice(r, c, [&](int v) { return ((usable >> v) & 1u) != 0; });
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("cls")
    (d / "s.cpp").write_text(SHIM)
    so = str(d / "s.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "s.cpp"),
                    "-o", so], check=True)
    lib = ct.CDLL(so)
    lib.cls.argtypes = [ct.c_longlong, ct.c_int, ct.c_int]
    return lib


@pytest.mark.parametrize("dirs", [1, 2, 24, 500])
def test_launches_of_few_tiles_and_of_more_share_no_class(lib, dirs):
    """Every launch size meets few classes, in order of size, and none on both sides of 16 tiles per
    SM, where the cooperative sweeps stop being candidates."""
    sms = 152
    seen = {True: [], False: []}
    for tiles in sorted({t + d for t in (1 << k for k in range(28)) for d in (-1, 0, 1) if t + d > 0} |
                        {16 * sms, 16 * sms + 1, 64 * sms, 64 * sms + 1}):
        few = tiles <= 16 * sms
        c = lib.cls(tiles * dirs, int(few), sms)
        assert 0 <= c < lib.classes()
        if not seen[few] or seen[few][-1] != c:
            seen[few].append(c)
    assert not set(seen[True]) & set(seen[False])
    assert seen[True] == sorted(seen[True]) and seen[False] == sorted(seen[False])
    assert len(seen[True]) <= 8 and len(seen[False]) <= 2


def test_the_nearest_usable_choice_is_kept(lib):
    row = (ct.c_int * 10)(-1, 3, -1, -1, 7, -1, -1, -1, 2, -1)
    every = 0xffffffff
    assert [lib.kept(row, c, every) for c in range(10)] == [3, 3, 3, 7, 7, 7, 7, 2, 2, 2]
    no7 = every & ~(1 << 7)  # a choice this launch cannot run is passed over, not kept
    assert [lib.kept(row, c, no7) for c in range(10)] == [3, 3, 3, 3, 3, 2, 2, 2, 2, 2]
    assert lib.kept(row, 4, 0) == -1
    assert lib.kept((ct.c_int * 10)(*[-1] * 10), 4, every) == -1
