"""The tensor-map cache of a suite (tealeaf_b200/csrc/tmacache.hpp), compiled
for the host: a launch looks up the maps its kernel takes, up to nine, before it
copies any, so none of them may be given up by the launch's later lookups. A
chunk's own arrays and the refinement's in both precisions come to 50 maps
against 48 entries."""
import ctypes as C
import random
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]

SOURCE = """
#include "tmacache.hpp"
struct alignas(64) Map { long key; };
static tl::TmaCache<Map, %d> cache;
static int encoded = 0;
// Looks up n keys (array = key, kind = key modulo 7) as one launch does; the
// number whose map, read afterwards, is another one's.
extern "C" int launch(const long* keys, int n)
{
    const Map* m[16];
    int wrong = 0;
    for (int i = 0; i < n; ++i)
        m[i] = cache.lookup((const void*)keys[i], (int)(keys[i] %% 7), [&](Map* q) {
            q->key = keys[i];
            ++encoded;
            return keys[i] >= 0;
        });
    for (int i = 0; i < n; ++i) wrong += (keys[i] >= 0 ? !m[i] || m[i]->key != keys[i] : m[i] != nullptr);
    return wrong;
}
extern "C" int encodings() { return encoded; }
"""


def _build(tmp_path, entries):
    src, lib = tmp_path / "cache.cpp", tmp_path / ("cache%d.so" % entries)
    src.write_text(SOURCE % entries)
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([cxx, "-std=c++17", "-shared", "-fPIC", "-I%s" % (REPO / "tealeaf_b200" / "csrc"), str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    return C.CDLL(str(lib))


def _launch(lib, keys):
    return lib.launch((C.c_long * len(keys))(*keys), len(keys))


@pytest.mark.parametrize("entries,keys", [(48, 40), (48, 48), (48, 50), (48, 200), (40, 41), (9, 30)])
def test_maps_of_a_launch_stay_its_own(tmp_path, entries, keys):
    lib = _build(tmp_path, entries)
    rng = random.Random(3)
    for _ in range(3000):
        assert _launch(lib, rng.sample(range(1, keys + 1), rng.randint(1, 9))) == 0
    if keys <= entries:
        assert lib.encodings() == keys   # and each is encoded once while all fit


def test_a_refused_encoding_gives_nothing_up(tmp_path):
    lib = _build(tmp_path, 9)
    assert _launch(lib, list(range(1, 10))) == 0
    assert _launch(lib, [-5, -6]) == 0
    assert _launch(lib, list(range(1, 10))) == 0
    assert lib.encodings() == 11
