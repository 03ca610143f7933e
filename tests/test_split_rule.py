"""The source splits of the potentials (csrc/splits.h), compiled on its own and called on the CPU."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dielectricbie.jl_b200", "csrc")
CHUNK = 128


@pytest.fixture(scope="module")
def splits(tmp_path_factory):
    d = tmp_path_factory.mktemp("splits")
    (d / "shim.cpp").write_text('#include "splits.h"\n'
                                'extern "C" int splits(int64_t n, int64_t t, int64_t s) { return bie::wave_splits(n, t, s); }')
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, str(d / "shim.cpp"), "-o",
                    str(d / "libsplits.so")], check=True)
    f = C.CDLL(str(d / "libsplits.so")).splits
    f.argtypes = [C.c_int64] * 3
    return f


@pytest.mark.parametrize("slots", [3 * 148, 4 * 148])
@pytest.mark.parametrize("n", [512, 2560, 18688, 42048])
def test_waves_are_full(splits, n, slots):
    """The slots' time is spent on sources: at least 3/4 of it from half a wave of tiles on, also where
    the tiles are a little more than half of the slots or a little more than all of them. Sources
    come in whole chunks, and n is at least 4 of them, so short sums cannot be cut finer."""
    chunks = -(-n // CHUNK)
    for tiles in list(range(slots // 2, 4 * slots, 7)) + [slots // 2 + 1, slots + 1, 313]:
        ns = splits(n, tiles, slots)
        assert 1 <= ns <= chunks
        waves = -(-tiles * ns // slots)
        busy = tiles * chunks / (slots * waves * -(-chunks // ns))
        one = tiles / (slots * -(-tiles // slots))  # the sources left whole
        assert busy >= (0.75 if chunks >= 20 else one), (tiles, ns, busy)


@pytest.mark.parametrize("tiles, n", [(1, 128), (1, 42048), (16, 42048), (7, 1000), (100000, 5000)])
def test_every_split_has_sources(splits, tiles, n):
    chunks = -(-n // CHUNK)
    for slots in (1, 444, 592):
        ns = splits(n, tiles, slots)
        per = -(-(-(-n // ns)) // CHUNK)  # the kernel's chunks per split
        assert 1 <= ns <= chunks and (ns - 1) * per < chunks
