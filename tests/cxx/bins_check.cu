// Host check of the cell sort's index arithmetic (psph_bins.cuh) up to the
// largest grid an upload accepts: bins and scan positions against 64-bit
// integers, over every split, the last cells and the last scan blocks. Prints
// the mismatch count and exits non-zero on any.
#include <cstdio>

#include "psph_bins.cuh"

using namespace psph;
typedef long long ll;

static ll bad = 0, checked = 0;
static void same(ll got, ll want, const char* what) {
  ++checked;
  if (got == want) return;
  if (bad < 10) printf("%s: %lld, not %lld\n", what, got, want);
  ++bad;
}

int main() {
  const ll cells[] = {1, 2, 1000, kMaxCells / 2 - 1, kMaxCells / 2, kMaxCells - 1, kMaxCells};
  for (ll nc : cells)
    for (int xs = 1; xs <= kMaxXsub; ++xs) {
      const ll bins = 2 * nc * xs, len = bins + 2;
      same(sort_bin((int)nc, xs, 0), bins, "bins");
      for (ll c = nc > 3 ? nc - 3 : 0; c < nc; ++c)
        for (int s = 0; s <= xs; ++s) {
          const unsigned b = sort_bin((int)c, xs, s);
          same(b, 2 * (c * xs + s), "bin");
          if (b < sort_bin((int)nc, xs, 0)) same(b / sort_bin(1, xs, 0), c + (s == xs), "cell of a bin");
        }
      const ll blocks = (len + kScanBlock - 1) / kScanBlock;
      same(scan_blocks_for((unsigned)len), blocks, "blocks");
      for (ll b = blocks > 3 ? blocks - 3 : 0; b < blocks; ++b)
        for (unsigned t = 0; t < 1024; ++t) {
          const unsigned first = scan_first((unsigned)b, t);
          same(first, b * kScanBlock + (ll)t * kScanPer, "first");
          same(scan_full(first, kScanPer, (unsigned)len), (ll)first + kScanPer <= len, "whole group of 8");
          same(scan_full(first, 4, (unsigned)len), (ll)first + 4 <= len, "whole group of 4");
        }
    }
  printf("checked %lld mismatches %lld\n", checked, bad);
  return bad ? 1 : 0;
}
