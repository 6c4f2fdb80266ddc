// Host BLAKE3 compressions (host_blake3.h): one, and eight at a time in the
// lanes of the compiler's vector types.
#include "host_blake3.h"

namespace hb3 {

void compress(const uint32_t cv[8], const uint32_t m[16], uint64_t ctr, uint32_t len, uint32_t flags,
              uint32_t out[16]) {
  uint32_t v[16] = {cv[0], cv[1], cv[2], cv[3], cv[4], cv[5], cv[6], cv[7],
                    IV[0], IV[1], IV[2], IV[3], (uint32_t)ctr, (uint32_t)(ctr >> 32), len, flags};
  rounds(v, m);
  for (int i = 0; i < 8; i++) {
    const uint32_t c = cv[i];  // out may be cv
    out[i] = v[i] ^ v[i + 8];
    out[i + 8] = v[i + 8] ^ c;
  }
}

namespace {
typedef uint32_t Lanes __attribute__((vector_size(32)));
}

void compress_lanes8(uint32_t cv[8][8], const uint8_t* const p[8], uint32_t len, uint32_t flags) {
  Lanes m[16], v[16];
  uint32_t w[8][16];
  for (int k = 0; k < 8; k++) load_words(p[k], len, w[k]);
  for (int i = 0; i < 16; i++)
    for (int k = 0; k < 8; k++) m[i][k] = w[k][i];
  for (int i = 0; i < 8; i++)
    for (int k = 0; k < 8; k++) v[i][k] = cv[k][i];
  const Lanes zero = {};
  for (int i = 0; i < 4; i++) v[8 + i] = zero + IV[i];
  v[12] = v[13] = zero;
  v[14] = zero + len;
  v[15] = zero + flags;
  rounds(v, m);
  for (int i = 0; i < 8; i++) {
    const Lanes c = v[i] ^ v[i + 8];
    for (int k = 0; k < 8; k++) cv[k][i] = c[k];
  }
}

}  // namespace hb3
