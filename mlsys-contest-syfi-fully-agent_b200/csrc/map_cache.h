// Host-side cache of encoded tensor maps.  A map is a pure function of its key (address, extents, strides, box), so an
// entry never goes stale; encoding one again costs about a microsecond of host time.
//
// Set-associative: a lookup hashes the key and compares at most kWays of them, a new map replaces the oldest of its set.
// Sized for a process that owns all eight shards of a layer: a call takes ten maps (two weight tensors, four token boxes
// of each GEMM's operand) whose keys hold the shard's weights and, through the row capacity, its batch size, so a pass
// over the layer uses 80 in a fixed order, and a few batch sizes stay side by side in 512.  (A first-in-first-out table
// of 64 entries, searched linearly, missed on every one of the 80.)  Not synchronised: the caller holds a lock.
#pragma once
#include <stdint.h>

namespace moe {

struct MapKey {
  const void* ptr;
  uint32_t rank;
  uint64_t dims[4];
  uint64_t strides[3];
  uint32_t box[4];
  bool operator==(const MapKey& o) const {
    if (ptr != o.ptr || rank != o.rank) return false;
    for (uint32_t i = 0; i < rank; ++i)
      if (dims[i] != o.dims[i] || box[i] != o.box[i]) return false;
    for (uint32_t i = 0; i + 1 < rank; ++i)
      if (strides[i] != o.strides[i]) return false;
    return true;
  }
  uint64_t hash() const {
    uint64_t h = reinterpret_cast<uintptr_t>(ptr);
    auto mix = [&](uint64_t v) {       // multiply and fold, one round per field
      h = (h ^ v) * 0x9E3779B97F4A7C15ull;
      h ^= h >> 32;
    };
    mix(rank);
    for (uint32_t i = 0; i < rank; ++i) { mix(dims[i]); mix(box[i]); }
    for (uint32_t i = 0; i + 1 < rank; ++i) mix(strides[i]);
    return h;
  }
};

template <class Map>
class MapCache {
 public:
  static constexpr int kSets = 64, kWays = 8;
  bool find(const MapKey& key, Map* out) const {
    const Set& s = sets_[key.hash() % kSets];
    for (int w = 0; w < s.used; ++w)
      if (s.key[w] == key) {
        *out = s.map[w];
        return true;
      }
    return false;
  }
  void insert(const MapKey& key, const Map& map) {
    Set& s = sets_[key.hash() % kSets];
    const int w = s.next;
    s.key[w] = key;
    s.map[w] = map;
    s.next = (w + 1) % kWays;
    if (s.used < kWays) ++s.used;
  }

 private:
  struct Set {
    Map map[kWays];
    MapKey key[kWays];
    int used = 0, next = 0;
  };
  Set sets_[kSets];
};

}  // namespace moe
