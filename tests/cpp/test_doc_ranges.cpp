// Host-side checks of the document ranges that decide which tiles the attention backward visits (csrc/tile_math.h), built
// with -fsanitize=address,undefined by tests/test_doc_ranges_host.py.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <random>
#include <vector>

#include "tile_math.h"

using namespace kf::tilemath;

static int failures = 0;
#define CHECK(cond)                                                                 \
  do {                                                                              \
    if (!(cond)) {                                                                  \
      std::fprintf(stderr, "%s:%d: check failed: %s\n", __FILE__, __LINE__, #cond); \
      ++failures;                                                                   \
    }                                                                               \
  } while (0)

constexpr int Q = 64, K = 128;  // positions of a query tile and of a key tile of the backward

static IdRange range_of(const std::vector<int>& ids, int first, int n) {
  IdRange r{INT_MAX, INT_MIN};
  for (int i = first; i < std::min<int>(first + n, int(ids.size())); ++i) r = {std::min(r.lo, ids[i]), std::max(r.hi, ids[i])};
  return r;
}

// Query tiles the key tiles visit; every tile with a visible pair is among them, none lies above the diagonal.
static int walked(const std::vector<int>& ids, bool causal) {
  const int s = int(ids.size()), nq = (s + Q - 1) / Q, nk = (s + K - 1) / K;
  int count = 0;
  for (int kt = 0; kt < nk; ++kt) {
    const int first = causal ? std::min(nq, kt * K / Q) : 0;
    const IdRange own = range_of(ids, kt * K, K);
    for (int j = 0; j < nq; ++j) {
      const bool on = query_tile_walked(j, first, range_of(ids, j * Q, Q), own);
      count += on;
      CHECK(!on || j >= first);
      bool visible = false;
      for (int q = j * Q; q < std::min(s, (j + 1) * Q) && !visible; ++q)
        for (int k = kt * K; k < std::min(s, (kt + 1) * K) && !visible; ++k) visible = ids[q] == ids[k] && (!causal || k <= q);
      CHECK(on || !visible);
    }
  }
  return count;
}

// first id, positions per document, documents, then `pad` positions with id `pad_id`
static std::vector<int> packed(int first, int len, int docs, int pad, int pad_id) {
  std::vector<int> v;
  for (int d = 0; d < docs; ++d) v.insert(v.end(), len, first + d);
  v.insert(v.end(), pad, pad_id);
  return v;
}

int main() {
  // adding the same number to every id changes nothing, also where the ids reach across zero
  for (int shift : {-9, -8, -1, 0, 1, 5}) CHECK(walked(packed(shift, 512, 8, 0, 0), true) == walked(packed(100, 512, 8, 0, 0), true));
  // documents 1..8 and padding with id 0: as many tiles as with every id moved away from zero
  CHECK(walked(packed(1, 450, 8, 496, 0), true) == walked(packed(101, 450, 8, 496, 100), true));
  // a key tile that holds ids on both sides of zero visits no tile above the diagonal: 64 query tiles, 32 key tiles, 2 each
  std::vector<int> zigzag(4096);
  for (int i = 0; i < 4096; ++i) zigzag[i] = i & 1;
  CHECK(walked(zigzag, true) == 32 * 33);
  CHECK(walked(zigzag, false) == 32 * 64);
  // one document: the causal triangle; a document per tile pair: the diagonal alone
  CHECK(walked(packed(0, 4096, 1, 0, 0), true) == 32 * 33);
  CHECK(walked(packed(-16, 128, 32, 0, 0), true) == 32 * 2);
  std::mt19937 rng(1);
  for (int n : {1, 63, 64, 65, 129, 700, 1000}) {
    std::vector<int> v(n);
    for (int& x : v) x = int(rng() % 9) - 4;
    walked(v, true);
    walked(v, false);
    for (int& x : v) x = (rng() & 1) ? INT_MAX : INT_MIN;
    walked(v, true);
  }
  if (failures) {
    std::fprintf(stderr, "%d check(s) failed\n", failures);
    return 1;
  }
  std::puts("doc_ranges: all checks passed");
  return 0;
}
