// The look-back words of the single-pass scans and sorts on the CPU: where
// the two kinds lie in an area, that no word a scan leaves can be read as a
// current one by a sort on the same area, in whatever order operations with
// whatever sums alternate, and the range of the sums that a scan's word carries.
#include <cstdio>
#include <cstring>
#include <vector>

#include "lookback.cuh"

using namespace dcsr;

#define CHECK(c)                                                      \
  do {                                                                \
    if (!(c)) {                                                       \
      fprintf(stderr, "line %d: %s\n", __LINE__, #c);                 \
      return 1;                                                       \
    }                                                                 \
  } while (0)

// A sort's test of a word at epoch e (k_radix_onesweep).
static bool sort_takes(unsigned long long word, unsigned long long e) {
  const unsigned tag2 = (unsigned)(e & LB_EMASK) << 2;
  return (unsigned)(word >> 32) - tag2 - 1u < 2u;
}

int main() {
  for (size_t slots : {2, 1024, 1026, 65536}) {
    std::vector<unsigned long long> mem(lb_bytes(slots) / 8 + 2);
    unsigned char *base = (unsigned char *)(((uintptr_t)mem.data() + 15) / 16 * 16);
    Lookback lb;
    std::memset(&lb, 0, sizeof(lb));
    lb_parts(base, slots, &lb);
    CHECK((unsigned char *)lb.flag == base + LB_HEADER);
    CHECK((uintptr_t)lb.scan % 16 == 0);
    CHECK(lb.scan >= lb.flag + slots && (unsigned char *)(lb.scan + slots) <= base + lb_bytes(slots));
    // every word of the scans' area written, with sums that look like tags of
    // the epochs to come: the sort reads none of them as its own
    for (unsigned long long e = 1; e < 40; e++) {
      for (size_t t = 0; t < slots / LB_SCAN_WORDS; t++) {
        const long long v3[3] = {(long long)t, (long long)(4 * (e + 1) + 1 + t % 2), 7};
        const long long v1[1] = {(long long)((4 * (e + 1) + 2) << 32)};
        const LbWord w = t % 3 ? lb_word<3>(e, 2, v3) : lb_word<1>(e, 2, v1);
        std::memcpy(lb.scan + LB_SCAN_WORDS * t, &w, sizeof(w));
      }
      for (size_t i = 0; i < slots; i++) CHECK(!sort_takes(lb.flag[i], e + 1));
    }
  }
  // what a word carries: a sum of 64 bits; sums of 64 and of 32; three of 32
  const long long big[] = {0, 1, 65535ll << 32, 1ll << 48, (1ll << 48) + 12345, 1ll << 61, INT64_MAX};
  const long long small[] = {0, 1, 65536, 0x7fffffffll, 0xffffffffll};
  for (unsigned long long e : {1ull, 77ull, LB_EMASK}) {
    for (long long a : big) {
      const long long v1[1] = {a};
      CHECK(lb_sum<1>(lb_word<1>(e, 1, v1), 0) == a);
      for (long long b : small) {
        const long long v2[2] = {a, b};
        const LbWord w = lb_word<2>(e, 2, v2);
        CHECK(lb_sum<2>(w, 0) == a && lb_sum<2>(w, 1) == b && w.hi >> 32 == ((e << 2) | 2));
      }
    }
    for (long long a : small)
      for (long long b : small) {
        const long long v3[3] = {a, b, a};
        const LbWord w = lb_word<3>(e, 1, v3);
        CHECK(lb_sum<3>(w, 0) == a && lb_sum<3>(w, 1) == b && lb_sum<3>(w, 2) == a && w.hi >> 32 == ((e << 2) | 1));
      }
  }
  printf("ok\n");
  return 0;
}
