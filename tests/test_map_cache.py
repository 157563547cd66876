"""CPU test of the tensor-map cache (csrc/map_cache.h): what a repeated pass of the eight-shard layer has to encode."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>
#include "map_cache.h"
using namespace moe;
struct Map { uint64_t tag[16]; };
static MapCache<Map> cache;
static std::vector<MapKey> keys;
static int encoded;
// the map of `key`, as the launcher gets it; its tag is the key's ordinal, so that a wrong hit shows
static bool get(const MapKey& key) {
  size_t id = 0;
  while (id < keys.size() && !(keys[id] == key)) ++id;
  if (id == keys.size()) keys.push_back(key);
  Map m{};
  if (!cache.find(key, &m)) { ++encoded; m.tag[0] = id; cache.insert(key, m); }
  return m.tag[0] == id;
}
static MapKey key3(uint64_t ptr, uint64_t rows, uint64_t K, uint32_t box_rows, uint32_t kps) {
  MapKey k{};
  k.ptr = reinterpret_cast<const void*>(ptr); k.rank = 3;
  k.dims[0] = 128; k.dims[1] = rows; k.dims[2] = K / 128; k.strides[0] = K; k.strides[1] = 128;
  k.box[0] = 128; k.box[1] = box_rows; k.box[2] = kps;
  return k;
}
static MapKey key4(uint64_t ptr, uint64_t rows, uint32_t box_rows) {
  MapKey k{};
  k.ptr = reinterpret_cast<const void*>(ptr); k.rank = 4;
  k.dims[0] = 128; k.dims[1] = rows; k.dims[2] = 3; k.dims[3] = 16;
  k.strides[0] = 2048; k.strides[1] = rows * 2048; k.strides[2] = 128;
  k.box[0] = 128; k.box[1] = box_rows; k.box[2] = 1; k.box[3] = 1;
  return k;
}
// the ten maps of a large-batch call of every shard: own weights, one shared workspace, own row capacity
static bool pass(uint64_t weights, uint64_t ws, uint64_t rows0) {
  bool ok = true;
  for (uint64_t s = 0; s < 8; ++s) {
    const uint64_t rows = rows0 + 128 * s, w = weights + s * (1409286144ull + (2ull << 20));
    ok &= get(key3(w, 131072, 7168, 128, 1)) && get(key3(w + 939524096ull, 229376, 2048, 128, 1));
    for (uint32_t r = 32; r <= 128; r += 32)
      ok &= get(key3(ws + rows * 64, rows, 7168, r, 1)) && get(key4(ws + rows * 7400, rows, r));
  }
  return ok;
}
int main(int argc, char** argv) {
  const uint64_t seed = std::strtoull(argv[1], nullptr, 10), base = 0x7f0000000000ull + seed * 0x35600000ull;
  const int sizes = std::atoi(argv[2]);
  bool ok = true;
  for (int b = 0; b < sizes; ++b) ok &= pass(base, base + (1ull << 36), 8192 + 2048 * b);
  const int first = encoded;
  for (int b = 0; b < sizes; ++b) ok &= pass(base, base + (1ull << 36), 8192 + 2048 * b);
  std::printf("%d %d %d %zu\n", ok, first, encoded - first, keys.size());
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("map_cache")
    (d / "probe.cpp").write_text(PROBE)
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", os.path.join(ROOT, "mlsys-contest-syfi-fully-agent_b200", "csrc"),
                    "-o", str(d / "probe"), str(d / "probe.cpp")], check=True)
    return str(d / "probe")


@pytest.mark.parametrize("sizes", [1, 2])
def test_a_repeated_pass_of_eight_shards_encodes_nothing(probe, sizes):
    """Eight shards with ten maps each, at one and at two batch sizes, from several base addresses: the second time every
    map is found, and it is the map of its key."""
    for seed in range(20):
        out = subprocess.run([probe, str(seed), str(sizes)], check=True, capture_output=True, text=True).stdout.split()
        ok, first, again, keys = (int(x) for x in out)
        assert ok == 1 and keys == 16 + 64 * sizes
        assert first == keys and again == 0, (seed, out)


def test_more_maps_than_the_cache_holds(probe):
    """Far more maps than entries: old ones are replaced, and whatever is found is the map of its key."""
    ok, first, again, keys = (int(x) for x in subprocess.run([probe, "3", "40"], check=True, capture_output=True,
                                                             text=True).stdout.split())
    assert ok == 1 and keys == 16 + 64 * 40 and again > 0
