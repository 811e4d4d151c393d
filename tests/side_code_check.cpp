// Host check of the side-set codes that travel with the k-mers
// (cf1_common.cuh): contribution_code's byte equals contribution_sideset for
// 64- and 128-bit k-mers, every combination of neighbours, and k-mers whose
// next k-mer is the same vertex (homopolymers, alternating repeats, k-mers
// that roll into their own reverse complement).  Prints "ok" and exits 0, or
// names the first failure and exits 1.
#include <cstdio>
#include <random>

#include "cf1_common.cuh"

using namespace cf1;

template <class K>
K kmer_of(std::mt19937_64 &rng, int k, int kind) {
  K fw{}, rc{};
  const uint32_t a = rng() & 3, b = rng() & 3;
  uint32_t half[64];
  for (int i = 0; i < k; i++) {
    uint32_t c = rng() & 3;
    if (kind == 1) c = a;                      // homopolymer
    if (kind == 2) c = i & 1 ? a : b;          // dinucleotide repeat
    if (kind == 3 && i > k / 2) c = 3 - half[k - i];  // first base, then a reverse palindrome
    half[i] = c;
    KOps<K>::roll(fw, rc, c, k);
  }
  return fw;
}

template <class K>
int check(int k) {
  std::mt19937_64 rng(k);
  uint64_t loops = 0;
  for (int it = 0; it < 60000; it++) {
    const K fw = kmer_of<K>(rng, k, it & 3), rc = KOps<K>::rc(fw, k);
    for (uint32_t prev = 0; prev < 4; prev++)
      for (uint32_t next = 0; next < 4; next++)
        for (int has = 0; has < 4; has++) {
          const bool hp = has & 1, hn = has & 2;
          K nf = fw, nr = rc;
          KOps<K>::roll(nf, nr, next, k);
          loops += kmin(nf, nr) == kmin(fw, rc);
          const uint32_t want = contribution_sideset(fw, rc, hp, prev, hn, next, k);
          const uint32_t code = contribution_code(fw, rc, nf, hp ? prev : 4u, hn, next);
          if (code >= 64 || pay_byte(code) != want) {
            std::printf("k=%d prev=%u next=%u has=%d: code %u gives %02x, not %02x\n", k, prev, next, has, code,
                        pay_byte(code), want);
            return 1;
          }
        }
  }
  if (!loops) std::printf("k=%d: no self loop among the k-mers\n", k);
  return loops ? 0 : 1;
}

int main() {
  for (int k : {1, 3, 5, 15, 21, 31})
    if (check<uint64_t>(k)) return 1;
  for (int k : {33, 45, 63})
    if (check<Key2>(k)) return 1;
  std::printf("ok\n");
  return 0;
}
