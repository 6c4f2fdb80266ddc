// Host BLAKE3 (public specification) for the Fiat-Shamir transcript and the
// statement digest. Incremental chunk state plus chaining-value stack; the
// root output is extendable (XOF). Matches the device compression in
// blake3.cuh word for word.
#pragma once
#include <array>
#include <cstdint>
#include <cstring>
#include <vector>

namespace hb3 {

static constexpr uint32_t IV[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a,
                                   0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
enum : uint32_t { CHUNK_START = 1, CHUNK_END = 2, PARENT = 4, ROOT = 8 };

// The message word that column/diagonal step i of round r takes: the BLAKE3
// permutation applied r times.
constexpr int kPerm[16] = {2, 6, 3, 10, 7, 0, 4, 13, 1, 11, 12, 5, 9, 14, 15, 8};
constexpr int msg_index(int r, int i) { return r == 0 ? i : msg_index(r - 1, kPerm[i]); }

// One round with its message order fixed at compile time: the sixteen state
// words stay in registers and the schedule costs no moves (a transcript's
// samples are chains of compressions: 650 ns a sample with the message permuted
// in memory every round, 350 ns so, 75 ns a compression, on a Grace core).
template <int R, class W>
inline __attribute__((always_inline)) void round_fn(W v[16], const W* m) {
#define HB3_G(a, b, c, d, i)                                                             \
  v[a] += v[b] + m[msg_index(R, i)];     v[d] ^= v[a]; v[d] = (v[d] >> 16) | (v[d] << 16); \
  v[c] += v[d];                          v[b] ^= v[c]; v[b] = (v[b] >> 12) | (v[b] << 20); \
  v[a] += v[b] + m[msg_index(R, i + 1)]; v[d] ^= v[a]; v[d] = (v[d] >> 8) | (v[d] << 24);  \
  v[c] += v[d];                          v[b] ^= v[c]; v[b] = (v[b] >> 7) | (v[b] << 25);
  HB3_G(0, 4, 8, 12, 0)
  HB3_G(1, 5, 9, 13, 2)
  HB3_G(2, 6, 10, 14, 4)
  HB3_G(3, 7, 11, 15, 6)
  HB3_G(0, 5, 10, 15, 8)
  HB3_G(1, 6, 11, 12, 10)
  HB3_G(2, 7, 8, 13, 12)
  HB3_G(3, 4, 9, 14, 14)
#undef HB3_G
}
template <class W>
inline __attribute__((always_inline)) void rounds(W v[16], const W* m) {
  round_fn<0>(v, m);
  round_fn<1>(v, m);
  round_fn<2>(v, m);
  round_fn<3>(v, m);
  round_fn<4>(v, m);
  round_fn<5>(v, m);
  round_fn<6>(v, m);
}

// (host_hash.cpp, so that the host compiler alone sees the unrolled rounds)
void compress(const uint32_t cv[8], const uint32_t m[16], uint64_t ctr, uint32_t len, uint32_t flags,
              uint32_t out[16]);

// Eight independent chaining values at a time, one per vector lane, with a
// zero counter: cv[k] = compress(cv[k], block k of 64 bytes at p[k], len, flags)
// (Merkle leaves and parents of one level; 51 ns each on a Grace core).
void compress_lanes8(uint32_t cv[8][8], const uint8_t* const p[8], uint32_t len, uint32_t flags);

inline void load_words(const uint8_t* b, size_t n, uint32_t w[16]) {  // little-endian hosts
  if (n < 64) memset(w, 0, 64);
  memcpy(w, b, n);
}

class Hasher {
 public:
  Hasher() { memcpy(cv_, IV, 32); }

  void update(const void* data, size_t n) {
    const uint8_t* p = (const uint8_t*)data;
    while (n) {
      if (buf_len_ == 64 && blocks_ == 15) close_chunk();
      if (buf_len_ == 64) {
        uint32_t w[16], o[16];
        load_words(buf_, 64, w);
        compress(cv_, w, chunk_, 64, blocks_ == 0 ? CHUNK_START : 0, o);
        memcpy(cv_, o, 32);
        blocks_++;
        buf_len_ = 0;
      }
      size_t take = 64 - buf_len_;
      if (take > n) take = n;
      memcpy(buf_ + buf_len_, p, take);
      buf_len_ += take;
      p += take;
      n -= take;
    }
  }

  // Root output bytes (XOF) of the current state; the state is unchanged.
  void xof(uint8_t* out, size_t n) const {
    Node o = root_node();
    for (uint64_t ctr = 0; n; ctr++) {
      uint32_t w[16];
      compress(o.cv, o.block, ctr, o.len, o.flags | ROOT, w);
      size_t take = n < 64 ? n : 64;
      memcpy(out, w, take);  // little-endian host
      out += take;
      n -= take;
    }
  }
  void finalize(uint8_t out[32]) const { xof(out, 32); }

 private:
  struct Node {
    uint32_t cv[8], block[16];
    uint64_t ctr;
    uint32_t len, flags;
  };
  void close_chunk() {
    uint32_t w[16], o[16];
    load_words(buf_, 64, w);
    compress(cv_, w, chunk_, 64, CHUNK_END, o);
    std::array<uint32_t, 8> ncv;
    memcpy(ncv.data(), o, 32);
    for (uint64_t total = chunk_ + 1; (total & 1) == 0; total >>= 1) {
      uint32_t blk[16];
      memcpy(blk, stack_.back().data(), 32);
      memcpy(blk + 8, ncv.data(), 32);
      stack_.pop_back();
      compress(IV, blk, 0, 64, PARENT, o);
      memcpy(ncv.data(), o, 32);
    }
    stack_.push_back(ncv);
    chunk_++;
    memcpy(cv_, IV, 32);
    blocks_ = 0;
    buf_len_ = 0;
  }
  Node root_node() const {
    Node o;
    memcpy(o.cv, cv_, 32);
    load_words(buf_, buf_len_, o.block);
    o.ctr = chunk_;
    o.len = (uint32_t)buf_len_;
    o.flags = CHUNK_END | (blocks_ == 0 ? CHUNK_START : 0);
    for (size_t i = stack_.size(); i-- > 0;) {
      uint32_t w[16];
      compress(o.cv, o.block, o.ctr, o.len, o.flags, w);
      Node p;
      memcpy(p.cv, IV, 32);
      memcpy(p.block, stack_[i].data(), 32);
      memcpy(p.block + 8, w, 32);
      p.ctr = 0;
      p.len = 64;
      p.flags = PARENT;
      o = p;
    }
    return o;
  }

  uint32_t cv_[8];
  uint8_t buf_[64];
  size_t buf_len_ = 0, blocks_ = 0;
  uint64_t chunk_ = 0;
  std::vector<std::array<uint32_t, 8>> stack_;
};

}  // namespace hb3
