// Host check of the side-set codes that travel with the k-mers
// (cf1_common.cuh): contribution_code's byte equals the byte computed side by side for
// 64- and 128-bit k-mers, every combination of neighbours, and k-mers whose
// next k-mer is the same vertex (homopolymers, alternating repeats, k-mers
// that roll into their own reverse complement).  Prints "ok" and exits 0, or
// names the first failure and exits 1.
#include <cstdio>
#include <random>

#include "cf1_common.cuh"

using namespace cf1;

// sideset_lookup(contribution(...)) computed directly: the side-set byte of
// one occurrence (front nibble low, back nibble high; M = 0xF), from what it
// depends on: whether the k-mer is read forward (fwd), whether it has a base
// before / after it (and which), whether the next k-mer is the same vertex
// (next_same) and, if so, the same oriented k-mer (next_same_fw).  prev is
// not read without has_prev, nor next, next_same, next_same_fw without
// has_next.
uint32_t sideset_byte(bool fwd, bool has_prev, uint32_t prev, bool has_next, uint32_t next, bool next_same,
                             bool next_same_fw) {
  if (!has_prev && !has_next) return 0xFFu;
  const uint32_t cp = side_code(prev), cpc = side_code(3 - prev);
  const uint32_t right = fwd ? (cp | 0xF0u) : (0x0Fu | (cpc << 4));
  if (!has_next) return right;
  if (next_same) return (!has_prev || next_same_fw) ? 0xFFu : right;
  const uint32_t cn = side_code(next), cnc = side_code(3 - next);
  if (!has_prev) return fwd ? (0x0Fu | (cn << 4)) : (cnc | 0xF0u);
  return fwd ? (cp | (cn << 4)) : (cnc | (cpc << 4));
}

// The same from the k-mer's forward and reverse-complement values and the
// next k-mer's (nf, nr: the k-mer rolled by `next`), which a caller walking
// the sequence has already; with !has_next nf and nr are not read.
template <class KeyT>
uint32_t contribution_sideset_rolled(KeyT fw, KeyT rcv, KeyT nf, KeyT nr, bool has_prev, uint32_t prev,
                                            bool has_next, uint32_t next) {
  const KeyT can = kmin(fw, rcv);
  return sideset_byte(fw == can, has_prev, prev, has_next, next, has_next && kmin(nf, nr) == can,
                      has_next && nf == fw);
}

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
          const uint32_t want = contribution_sideset_rolled(fw, rc, nf, nr, hp, prev, hn, next);
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
