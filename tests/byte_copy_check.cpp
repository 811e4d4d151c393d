// Host check of byte_copy (cf1_common.cuh): the copy it lays out, carried out
// as the kernels do, writes every byte once and reads no aligned source word
// that reaches past the source.
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <vector>

#include "cf1_common.cuh"

using namespace cf1;

static bool check(uint32_t doff, uint32_t soff, uint32_t n) {
  alignas(8) uint8_t sb[128], db[128];
  for (uint32_t i = 0; i < sizeof(sb); i++) sb[i] = (uint8_t)(i * 37 + 11), db[i] = 0xEE;
  uint8_t *dst = db + 8 + doff;
  const uint8_t *src = sb + 8 + soff;
  const ByteCopy c = byte_copy((uintptr_t)dst, (uintptr_t)src, n);
  if (c.head > n || c.head + 4ull * c.words > n) return false;
  if (c.words && (((uintptr_t)dst + c.head) & 3)) return false;
  const uint32_t rest = n - c.head - 4 * c.words;
  if (rest > 6) return false;  // copied by the first threads of a warp
  std::vector<int> wrote(n, 0);
  for (uint32_t i = 0; i < c.head; i++) dst[i] = src[i], wrote[i]++;
  const uint8_t *w = src + c.head - c.shift / 8;
  if (c.words && ((uintptr_t)w & 3)) return false;
  for (uint32_t i = 0; i < c.words; i++) {
    if (w + 4 * i + (c.shift ? 8 : 4) > src + n) return false;  // reads past the source
    if (w + 4 * i + 4 <= src) return false;                    // or a word wholly before it
    uint32_t a, b = 0;
    std::memcpy(&a, w + 4 * i, 4);
    if (c.shift) std::memcpy(&b, w + 4 * i + 4, 4);
    const uint32_t v = c.shift ? (a >> c.shift) | (b << (32 - c.shift)) : a;
    std::memcpy(dst + c.head + 4 * i, &v, 4);
    for (int j = 0; j < 4; j++) wrote[c.head + 4 * i + j]++;
  }
  for (uint32_t i = n - rest; i < n; i++) dst[i] = src[i], wrote[i]++;
  for (uint32_t i = 0; i < n; i++)
    if (dst[i] != src[i] || wrote[i] != 1) return false;
  return dst[-1] == 0xEE && dst[n] == 0xEE;
}

int main() {
  for (uint32_t d = 0; d < 4; d++)
    for (uint32_t s = 0; s < 4; s++)
      for (uint32_t n = 0; n <= 64; n++)
        if (!check(d, s, n)) {
          std::printf("dst %u src %u n %u\n", d, s, n);
          return 1;
        }
  std::puts("ok");
  return 0;
}
