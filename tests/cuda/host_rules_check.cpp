// Host check of the kernels' arithmetic rules (hsr_internal.h): prints one line per failure.
#include <cstdio>
#include <initializer_list>

#include "hsr_internal.h"

using namespace hsr;

static int failures = 0;
#define CHECK(c)                                        \
  do {                                                  \
    if (!(c)) {                                         \
      std::printf("line %d: %s\n", __LINE__, #c);       \
      failures++;                                       \
    }                                                   \
  } while (0)

// The shares of a list partition it, in order, whatever its length.
static void shares() {
  for (uint32_t parts : {4u, 8u})
    for (uint32_t n : {0u, 1u, 3u, 4u, 7u, 8u, 9u, 1000u, 1u << 29, (1u << 29) + 1u, 1u << 30, 0x7fffffffu, 0xfffffffeu}) {
      CHECK(share_begin(n, 0, parts) == 0u);
      CHECK(share_begin(n, parts, parts) == n);
      for (uint32_t k = 0; k < parts; k++) {
        const uint32_t b = share_begin(n, k, parts), e = share_begin(n, k + 1, parts);
        CHECK(b <= e && e - b <= n / parts + 1u);
      }
    }
}

// Every group of 32 records has its warps, whatever the grid, and each warp's step is a whole group.
static void sharers() {
  for (uint32_t warps : {1u, 2u, 8u, 15u, 16u, 17u, 40u, 9728u})
    for (uint32_t nrec : {0u, 1u, 31u, 32u, 33u, 100u, 5000u, 1u << 20, 0xfffff000u}) {
      const uint32_t parts = scatter_sharers(nrec, warps), groups = warps / parts;
      CHECK(parts >= 1u && parts <= kMaxSharers && groups >= 1u);
      CHECK(parts == 1u || groups * 32u >= nrec || parts * nrec <= warps * 32u);
    }
}

// Six draws into one 1280x720 target, five pixels to clear a pair and draw: what the five that do not
// clear leave empty is not to be cleared.  One draw of 15 pixels a pair: two blocks of three clear.
static void clears() {
  const size_t px = 1280 * 720, tiles = px / 64;
  const uint32_t empty = (uint32_t)(tiles / 2);
  CHECK(scatter_every(6 * empty, 8, clear_share(12 * px, 6 * px), (uint32_t)(px / 2 / 5)) == 2u);
  CHECK(scatter_every(empty, 8, clear_share(12 * px, px), (uint32_t)(px / 2 / 15)) == 3u);
  CHECK(scatter_every(empty, 8, clear_share(4 * px, px), (uint32_t)(px / 2 / 15)) == 2u);  // colour alone
  CHECK(clear_share(0, 0) == 0.f);
}

int main() {
  shares();
  sharers();
  clears();
  return failures != 0;
}
