// BLAKE3 R1CS witness generation: one thread per compression.
//
// Restates the witness of crates/flock-prover/src/r1cs_hashes/blake3.rs:965-1076
// and its packed (z, a, b) writer at :1124-1290 (r1cs_hashes/common.rs:85-101):
// per compression a 2^14-bit block in the layout of blake3.rs:107-231
//   [0,256) cv | [256,512) out_lo | 512 const | [513,1025) m | t_lo | t_hi |
//   block_len | flags | 56 G-blocks x 250 bits | [15153,15409) out_hi | zeros
// For a carry-only ADD x + y with cin = (x + y) ^ x ^ y, bits 0..30 hold
// z = (x^cin)&(y^cin), a = x^cin, b = y^cin; input and lin-id words hold
// z = a = value, b = all ones; the constant bit is (1,1,1); c = z.
// It also writes the lincheck byte stripe of crates/flock-core/src/lincheck.rs:88-110:
// byte (j/8)*2^14 + i has bit (j%8) = witness bit i of compression j.
//
// Threads run the data-independent BLAKE3 schedule in lockstep, so every lane
// completes witness word w at the same instruction. Completed 64-bit words are
// staged per warp in shared memory and written out 16 words at a time as
// 128-byte runs per compression; the stripe bytes of each group of eight
// compressions are produced from the same staging by bit transposes.
#include <cstdint>

#include "blake3.cuh"
#include "flock_internal.h"

namespace {

constexpr int STAGE_WORDS = 16;
constexpr int STAGE_STRIDE = STAGE_WORDS + 1;  // 64-bit words; avoids bank conflicts
constexpr int WARPS_PER_BLOCK = 4;
constexpr int KWORDS = 256;  // 64-bit words per compression block

struct WarpCtx {
  uint64_t* sz;  // [32][STAGE_STRIDE]
  uint64_t* sa;
  uint64_t* sb;
  uint64_t* gz;
  uint64_t* ga;
  uint64_t* gb;
  uint8_t* stripe;
  size_t warp_slot0;  // first compression slot of this warp
  int n_valid;        // valid lanes in this warp (slots < n_total)
  int lane;
};

// The stripe bytes of one witness word of eight compressions (rows): byte 8 p + i
// of the 64 is bit i of byte p of the rows, row r at bit r. Three rounds of bit
// exchanges between the rows' registers (row bit against bit index), after
// which row i holds the bytes of bit i, then 4 x 4 byte transposes.
// Gathering each byte of the rows by shifts and transposing 8 x 8 bits at a time
// cost several times the instructions: 2^17 slots of witness_kernel 203 -> 186 us,
// 0.86 of the measured HBM rate (199 -> 180 us, 0.89, on another GPU).
__device__ __forceinline__ void stripe_exchange(uint32_t& a, uint32_t& b, int k, uint32_t low) {
  const uint32_t t = ((a >> k) ^ b) & low;
  b ^= t;
  a ^= t << k;
}

__device__ __forceinline__ void stripe_bytes(const uint64_t* rows, uint4* out) {
#pragma unroll
  for (int h = 0; h < 2; h++) {  // bytes 0..3 and 4..7 of the words
    uint32_t v[8];
#pragma unroll
    for (int r = 0; r < 8; r++) v[r] = (uint32_t)(rows[r] >> (32 * h));
#pragma unroll
    for (int r = 0; r < 4; r++) stripe_exchange(v[r], v[r + 4], 4, 0x0F0F0F0Fu);
#pragma unroll
    for (int r = 0; r < 4; r++) stripe_exchange(v[r + (r & 2)], v[r + (r & 2) + 2], 2, 0x33333333u);
#pragma unroll
    for (int r = 0; r < 4; r++) stripe_exchange(v[2 * r], v[2 * r + 1], 1, 0x55555555u);
    uint32_t w[4][2];  // [byte][bits 0..3, 4..7]
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const uint32_t x0 = __byte_perm(v[4 * q], v[4 * q + 1], 0x5140), x1 = __byte_perm(v[4 * q], v[4 * q + 1], 0x7362);
      const uint32_t y0 = __byte_perm(v[4 * q + 2], v[4 * q + 3], 0x5140);
      const uint32_t y1 = __byte_perm(v[4 * q + 2], v[4 * q + 3], 0x7362);
      w[0][q] = __byte_perm(x0, y0, 0x5410);
      w[1][q] = __byte_perm(x0, y0, 0x7632);
      w[2][q] = __byte_perm(x1, y1, 0x5410);
      w[3][q] = __byte_perm(x1, y1, 0x7632);
    }
    out[2 * h] = make_uint4(w[0][0], w[0][1], w[1][0], w[1][1]);
    out[2 * h + 1] = make_uint4(w[2][0], w[2][1], w[3][0], w[3][1]);
  }
}

// Writes the 16 staged words (global word index w0..w0+15) of all lanes.
// (Scalar arguments, so the call passes them in registers; the context
// struct itself never has to live in memory.)
__device__ __noinline__ void flush_words(uint64_t* sz, uint64_t* gz, uint64_t* ga, uint64_t* gb, uint8_t* stripe,
                                        size_t warp_slot0, int n_valid, int lane, int w0) {
  struct {
    uint64_t *sz, *sa, *sb, *gz, *ga, *gb;
    uint8_t* stripe;
    size_t warp_slot0;
    int n_valid, lane;
  } c = {sz, sz + 32 * STAGE_STRIDE, sz + 64 * STAGE_STRIDE, gz, ga, gb, stripe, warp_slot0, n_valid, lane};
  __syncwarp();
  const int half = c.lane >> 4, j = c.lane & 15;
#pragma unroll 4
  for (int i = 0; i < 16; i++) {
    int comp = 2 * i + half;
    if (comp < c.n_valid) {
      size_t g = (c.warp_slot0 + comp) * KWORDS + w0 + j;
      c.gz[g] = c.sz[comp * STAGE_STRIDE + j];
      if (c.ga) {
        c.ga[g] = c.sa[comp * STAGE_STRIDE + j];
        c.gb[g] = c.sb[comp * STAGE_STRIDE + j];
      }
    }
  }
  if (c.stripe) {
    // 4 groups of 8 compressions x 16 words; two items per lane.
#pragma unroll
    for (int k = 0; k < 2; k++) {
      int item = c.lane + 32 * k;
      int grp = item >> 4, w = item & 15;
      if (8 * grp < c.n_valid) {
        uint64_t r8[8];
#pragma unroll
        for (int r = 0; r < 8; r++) r8[r] = c.sz[(8 * grp + r) * STAGE_STRIDE + w];
        size_t byte_idx = (c.warp_slot0 >> 3) + grp;
        uint4* dst = reinterpret_cast<uint4*>(c.stripe + byte_idx * (size_t)FLOCK_K + (size_t)(w0 + w) * 64);
        stripe_bytes(r8, dst);
      }
    }
  }
  __syncwarp();
}

struct Sink {
  uint64_t pz, pa, pb;
  int used;
  int word;
  __device__ __forceinline__ void emit(const WarpCtx& c, uint64_t z, uint64_t a, uint64_t b) {
    int j = word % STAGE_WORDS;
    c.sz[c.lane * STAGE_STRIDE + j] = z;
    c.sa[c.lane * STAGE_STRIDE + j] = a;
    c.sb[c.lane * STAGE_STRIDE + j] = b;
    word++;
    if (word % STAGE_WORDS == 0)
      flush_words(c.sz, c.gz, c.ga, c.gb, c.stripe, c.warp_slot0, c.n_valid, c.lane, word - STAGE_WORDS);
  }
  // Appends `width` bits (values already masked to width).
  __device__ __forceinline__ void push(const WarpCtx& c, uint32_t z, uint32_t a, uint32_t b, int width) {
    pz |= (uint64_t)z << used;
    pa |= (uint64_t)a << used;
    pb |= (uint64_t)b << used;
    if (used + width >= 64) {
      emit(c, pz, pa, pb);
      int sh = 64 - used;
      pz = sh >= 32 ? 0 : ((uint64_t)z >> sh);
      pa = sh >= 32 ? 0 : ((uint64_t)a >> sh);
      pb = sh >= 32 ? 0 : ((uint64_t)b >> sh);
      used = used + width - 64;
    } else {
      used += width;
    }
  }
  __device__ __forceinline__ void lin(const WarpCtx& c, uint32_t v) { push(c, v, v, 0xFFFFFFFFu, 32); }
  __device__ __forceinline__ uint32_t add(const WarpCtx& c, uint32_t x, uint32_t y) {
    uint32_t sum = x + y;
    uint32_t cin = sum ^ x ^ y;
    uint32_t l = (x ^ cin) & 0x7FFFFFFFu, r = (y ^ cin) & 0x7FFFFFFFu;
    push(c, l & r, l, r, 31);
    return sum;
  }
};

#define WG(LA, LB, LC, LD, R, S)                                        \
  {                                                                     \
    uint32_t a_ = s[LA], b_ = s[LB], c_ = s[LC], d_ = s[LD];            \
    uint32_t mx = mp[S], my = mp[S + 1];                                \
    uint32_t t0 = k.add(c, a_, b_);                                     \
    uint32_t a1 = k.add(c, t0, mx);                                     \
    uint32_t d1 = b3::rotr(d_ ^ a1, 16);                                \
    uint32_t c1 = k.add(c, c_, d1);                                     \
    uint32_t b1 = b3::rotr(b_ ^ c1, 12);                                \
    uint32_t t1 = k.add(c, a1, b1);                                     \
    uint32_t a2 = k.add(c, t1, my);                                     \
    uint32_t d2 = b3::rotr(d1 ^ a2, 8);                                 \
    uint32_t c2 = k.add(c, c1, d2);                                     \
    uint32_t bn = b3::rotr(b1 ^ c2, 7);                                 \
    k.lin(c, bn);                                                       \
    k.lin(c, d2);                                                       \
    s[LA] = a2; s[LB] = bn; s[LC] = c2; s[LD] = d2;                     \
  }

__global__ void __launch_bounds__(32 * WARPS_PER_BLOCK)
witness_kernel(const flock_compression* __restrict__ in, size_t n_in, size_t n_total, uint64_t* gz,
               uint64_t* ga, uint64_t* gb, uint8_t* stripe) {
  extern __shared__ uint64_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t slot = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t warp_slot0 = slot - lane;
  if (warp_slot0 >= n_total) return;
  WarpCtx c;
  uint64_t* base = smem + (size_t)warp * 3 * 32 * STAGE_STRIDE;
  c.sz = base;
  c.sa = base + 32 * STAGE_STRIDE;
  c.sb = base + 64 * STAGE_STRIDE;
  c.gz = gz; c.ga = ga; c.gb = gb; c.stripe = stripe;
  c.warp_slot0 = warp_slot0;
  size_t rem = n_total - warp_slot0;
  c.n_valid = rem >= 32 ? 32 : (int)rem;
  c.lane = lane;

  // Inputs: real compression, or the all-zero padding compression.
  uint32_t cv[8], m[16];
  uint64_t counter = 0;
  uint32_t blen = 0, flg = 0;
  if (slot < n_in) {
    const flock_compression& x = in[slot];
#pragma unroll
    for (int i = 0; i < 8; i++) cv[i] = x.cv[i];
#pragma unroll
    for (int i = 0; i < 16; i++) m[i] = x.m[i];
    counter = x.counter; blen = x.block_len; flg = x.flags;
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) cv[i] = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) m[i] = 0;
  }
  // out_lo sits before the G blocks in the layout: compute the output first.
  uint32_t out[16];
  b3::compress(cv, m, counter, blen, flg, out);

  Sink k{0, 0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 8; i++) k.lin(c, cv[i]);
#pragma unroll
  for (int i = 0; i < 8; i++) k.lin(c, out[i]);
  k.push(c, 1, 1, 1, 1);  // constant wire at bit 512
#pragma unroll
  for (int i = 0; i < 16; i++) k.lin(c, m[i]);
  uint32_t tlo = (uint32_t)counter, thi = (uint32_t)(counter >> 32);
  k.lin(c, tlo);
  k.lin(c, thi);
  k.lin(c, blen);
  k.lin(c, flg);
  uint32_t s[16] = {cv[0], cv[1], cv[2], cv[3], cv[4], cv[5], cv[6], cv[7],
                    b3::IV(0), b3::IV(1), b3::IV(2), b3::IV(3), tlo, thi, blen, flg};
  uint32_t mp[16];  // this round's message order
#pragma unroll
  for (int i = 0; i < 16; i++) mp[i] = m[i];
#pragma unroll
  for (int r = 0; r < 7; r++) {
    WG(0, 4, 8, 12, r, 0);
    WG(1, 5, 9, 13, r, 2);
    WG(2, 6, 10, 14, r, 4);
    WG(3, 7, 11, 15, r, 6);
    WG(0, 5, 10, 15, r, 8);
    WG(1, 6, 11, 12, r, 10);
    WG(2, 7, 8, 13, r, 12);
    WG(3, 4, 9, 14, r, 14);
    if (r < 6) b3::permute(mp);
  }
#pragma unroll
  for (int i = 0; i < 8; i++) k.lin(c, s[i + 8] ^ cv[i]);  // out_hi
  // Flush the partial word, then zero words up to the end of the block.
  k.emit(c, k.pz, k.pa, k.pb);
  while (k.word < KWORDS) k.emit(c, 0, 0, 0);
}

// ---- few compressions ------------------------------------------------------
//
// With a thread per compression a small batch is one thread's chain of about ten
// thousand instructions, unrolled and fetched once (60..70 us whatever the size). Here
// four lanes take a compression, a column (then diagonal) each: a G's 250
// witness bits are packed in registers, shifted to their place in the block and
// joined into the block's image in shared memory (the words a G shares with its
// neighbours by atomic ORs), the rounds in one loop body. The block then leaves
// in 16-byte vectors, the stripe bytes by the same transposes. 2^8
// compressions: 70 us through witness_kernel, 11 us so; 2^13: 61 us and 27 us;
// 2^14: 62 us and 46 us; 2^15: 84 us so (half of a block's threads wait while the
// rounds run, so the bandwidth-bound form wins beyond).
constexpr int WS_COMPS = 16, WS_THREADS = 128, WS_STRIDE = 512 + 4;  // 32-bit words of a block's image, padded
constexpr size_t WS_SMEM = ((size_t)3 * WS_COMPS * WS_STRIDE + WS_COMPS * 17) * 4;
constexpr size_t kSmallWitness = (size_t)1 << 14;  // slots
constexpr int kGBits = 250, kGFirst = 1153, kOutHi = 15153;

__constant__ uint8_t ws_msg[7][16] = {
    {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15}, {2, 6, 3, 10, 7, 0, 4, 13, 1, 11, 12, 5, 9, 14, 15, 8},
    {3, 4, 10, 12, 13, 2, 7, 14, 6, 5, 9, 0, 11, 15, 8, 1}, {10, 7, 12, 9, 14, 3, 13, 15, 4, 0, 11, 2, 5, 8, 1, 6},
    {12, 13, 9, 11, 15, 10, 14, 8, 7, 2, 5, 3, 0, 1, 6, 4}, {9, 14, 11, 5, 8, 12, 15, 1, 13, 3, 0, 10, 2, 6, 4, 7},
    {11, 15, 5, 0, 1, 9, 8, 6, 14, 10, 2, 12, 3, 4, 7, 13}};

// The 250 bits of one array of a G, 31 bits at a time.
struct GBits {
  uint32_t w[8];
  template <int AT>
  __device__ __forceinline__ void put(uint32_t v) {
    w[AT >> 5] |= v << (AT & 31);
    if constexpr ((AT & 31) != 0 && (AT >> 5) + 1 < 8) w[(AT >> 5) + 1] |= v >> (32 - (AT & 31));
  }
  // ORed into the image at bit `at`.
  __device__ __forceinline__ void store(uint32_t* img, int at) const {
    uint32_t* d = img + (at >> 5);
    const int sh = at & 31;
    atomicOr(d, w[0] << sh);
#pragma unroll
    for (int k = 1; k < 7; k++) d[k] = __funnelshift_l(w[k - 1], w[k], sh);
    atomicOr(d + 7, __funnelshift_l(w[6], w[7], sh));
    const uint32_t hi = __funnelshift_l(w[7], 0u, sh);
    if (hi) atomicOr(d + 8, hi);
  }
};

__device__ __forceinline__ void ws_or(uint32_t* img, int at, uint32_t v) {
  const int sh = at & 31;
  atomicOr(img + (at >> 5), v << sh);
  if (sh) atomicOr(img + (at >> 5) + 1, v >> (32 - sh));
}

template <int AT>
__device__ __forceinline__ uint32_t ws_add(uint32_t x, uint32_t y, GBits& z, GBits& a, GBits& b) {
  const uint32_t sum = x + y, cin = sum ^ x ^ y;
  const uint32_t l = (x ^ cin) & 0x7FFFFFFFu, r = (y ^ cin) & 0x7FFFFFFFu;
  z.put<AT>(l & r);
  a.put<AT>(l);
  b.put<AT>(r);
  return sum;
}

__global__ void __launch_bounds__(WS_THREADS)
witness_small_kernel(const flock_compression* __restrict__ in, size_t n_in, size_t n_total, uint64_t* gz, uint64_t* ga,
                     uint64_t* gb, uint8_t* stripe) {
  extern __shared__ __align__(16) uint32_t ws_smem[];
  uint32_t* img[3] = {ws_smem, ws_smem + WS_COMPS * WS_STRIDE, ws_smem + 2 * WS_COMPS * WS_STRIDE};  // z, a, b
  uint32_t* msgs = ws_smem + 3 * WS_COMPS * WS_STRIDE;
  const int t = threadIdx.x;
  const size_t slot0 = (size_t)blockIdx.x * WS_COMPS;
  const int n_valid = n_total - slot0 < WS_COMPS ? (int)(n_total - slot0) : WS_COMPS;
  for (int e = t; e < 3 * WS_COMPS * WS_STRIDE / 4; e += WS_THREADS)
    reinterpret_cast<uint4*>(ws_smem)[e] = make_uint4(0, 0, 0, 0);
  for (int e = t; e < WS_COMPS * 16; e += WS_THREADS) {
    const size_t slot = slot0 + (e >> 4);
    msgs[(e >> 4) * 17 + (e & 15)] = slot < n_in ? in[slot].m[e & 15] : 0u;
  }
  __syncthreads();
  if (t < 4 * WS_COMPS) {
    const int comp = t >> 2, q = t & 3;
    const size_t slot = slot0 + comp;
    uint32_t *z = img[0] + comp * WS_STRIDE, *ia = img[1] + comp * WS_STRIDE, *ib = img[2] + comp * WS_STRIDE;
    const uint32_t* m = msgs + comp * 17;
    uint32_t cv0 = 0, cv1 = 0, tail = 0;
    if (slot < n_in) {
      const flock_compression& x = in[slot];
      cv0 = x.cv[q];
      cv1 = x.cv[4 + q];
      tail = q == 0 ? (uint32_t)x.counter : q == 1 ? (uint32_t)(x.counter >> 32) : q == 2 ? x.block_len : x.flags;
    }
    uint32_t a = cv0, b = cv1, c = q == 0 ? b3::IV(0) : q == 1 ? b3::IV(1) : q == 2 ? b3::IV(2) : b3::IV(3), d = tail;
    // input words (z = a = value, b = all ones) and the constant bit
    z[q] = ia[q] = cv0;
    z[4 + q] = ia[4 + q] = cv1;
    if (q == 0) {
      atomicOr(&z[16], 1u);
      atomicOr(&ia[16], 1u);
      atomicOr(&ib[36], 1u);
    }
    for (int k = q; k < 36; k += 4) ib[k] = 0xFFFFFFFFu;
    for (int i = 4 * q; i < 4 * q + 4; i++) {
      ws_or(z, 513 + 32 * i, m[i]);
      ws_or(ia, 513 + 32 * i, m[i]);
    }
    ws_or(z, 1025 + 32 * q, tail);
    ws_or(ia, 1025 + 32 * q, tail);
#pragma unroll 1
    for (int h = 0; h < 14; h++) {  // half rounds: columns, then diagonals
      const bool diag = h & 1;
      if (diag) {
        b = __shfl_sync(0xffffffffu, b, q + 1, 4);
        c = __shfl_sync(0xffffffffu, c, q + 2, 4);
        d = __shfl_sync(0xffffffffu, d, q + 3, 4);
      }
      const int mi = (diag ? 8 : 0) + 2 * q;
      const uint32_t mx = m[ws_msg[h >> 1][mi]], my = m[ws_msg[h >> 1][mi + 1]];
      GBits gz_, ga_, gb_;
#pragma unroll
      for (int k = 0; k < 8; k++) gz_.w[k] = ga_.w[k] = gb_.w[k] = 0;
      const uint32_t t0 = ws_add<0>(a, b, gz_, ga_, gb_);
      const uint32_t a1 = ws_add<31>(t0, mx, gz_, ga_, gb_);
      const uint32_t d1 = b3::rotr(d ^ a1, 16);
      const uint32_t c1 = ws_add<62>(c, d1, gz_, ga_, gb_);
      const uint32_t b1 = b3::rotr(b ^ c1, 12);
      const uint32_t t1 = ws_add<93>(a1, b1, gz_, ga_, gb_);
      a = ws_add<124>(t1, my, gz_, ga_, gb_);
      d = b3::rotr(d1 ^ a, 8);
      c = ws_add<155>(c1, d, gz_, ga_, gb_);
      b = b3::rotr(b1 ^ c, 7);
      gz_.put<186>(b); ga_.put<186>(b); gb_.put<186>(0xFFFFFFFFu);
      gz_.put<218>(d); ga_.put<218>(d); gb_.put<218>(0xFFFFFFFFu);
      const int at = kGFirst + kGBits * (4 * h + q);
      gz_.store(z, at);
      ga_.store(ia, at);
      gb_.store(ib, at);
      if (diag) {
        b = __shfl_sync(0xffffffffu, b, q + 3, 4);
        c = __shfl_sync(0xffffffffu, c, q + 2, 4);
        d = __shfl_sync(0xffffffffu, d, q + 1, 4);
      }
    }
    z[8 + q] = ia[8 + q] = a ^ c;
    z[12 + q] = ia[12 + q] = b ^ d;
    ws_or(z, kOutHi + 32 * q, c ^ cv0);
    ws_or(ia, kOutHi + 32 * q, c ^ cv0);
    ws_or(ib, kOutHi + 32 * q, 0xFFFFFFFFu);
    ws_or(z, kOutHi + 128 + 32 * q, d ^ cv1);
    ws_or(ia, kOutHi + 128 + 32 * q, d ^ cv1);
    ws_or(ib, kOutHi + 128 + 32 * q, 0xFFFFFFFFu);
  }
  __syncthreads();
  uint64_t* out[3] = {gz, ga, gb};
  for (int k = 0; k < 3; k++) {
    if (!out[k]) continue;
    uint4* g = reinterpret_cast<uint4*>(out[k] + slot0 * KWORDS);
    for (int e = t; e < n_valid * 128; e += WS_THREADS)
      g[e] = *reinterpret_cast<const uint4*>(img[k] + (e >> 7) * WS_STRIDE + 4 * (e & 127));
  }
  if (stripe) {
    for (int item = t; item < (n_valid >> 3) * KWORDS; item += WS_THREADS) {
      const int grp = item / KWORDS, w = item % KWORDS;
      uint64_t r8[8];
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const uint2 v = *reinterpret_cast<const uint2*>(img[0] + (8 * grp + r) * WS_STRIDE + 2 * w);
        r8[r] = v.x | ((uint64_t)v.y << 32);
      }
      uint4* dst = reinterpret_cast<uint4*>(stripe + ((slot0 >> 3) + grp) * (size_t)FLOCK_K + (size_t)w * 64);
      stripe_bytes(r8, dst);
    }
  }
}

}  // namespace

int flock_launch_witness(const flock_compression* d_in, size_t n_in, int n_blocks_log, void* d_z, void* d_a,
                         void* d_b, void* d_stripe, cudaStream_t stream) {
  size_t n_total = (size_t)1 << n_blocks_log;
  if (n_in > n_total || n_blocks_log < 3) return FLOCK_ERR_SHAPE;
  if ((d_a == nullptr) != (d_b == nullptr)) return FLOCK_ERR_SHAPE;
  // (its 16-byte stores; witness_kernel stores z, a and b by 8 bytes)
  const bool aligned = (((uintptr_t)d_z | (uintptr_t)d_a | (uintptr_t)d_b) & 15) == 0;
  if (n_total <= kSmallWitness && aligned) {
    flock_once_per_device((const void*)witness_small_kernel, [] {
      cudaFuncSetAttribute(witness_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM);
    });
    witness_small_kernel<<<(unsigned)((n_total + WS_COMPS - 1) / WS_COMPS), WS_THREADS, WS_SMEM, stream>>>(
        d_in, n_in, n_total, (uint64_t*)d_z, (uint64_t*)d_a, (uint64_t*)d_b, (uint8_t*)d_stripe);
    flock_count_launch();
    return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
  }
  const int threads = 32 * WARPS_PER_BLOCK;
  size_t blocks = (n_total + threads - 1) / threads;
  size_t smem = (size_t)WARPS_PER_BLOCK * 3 * 32 * STAGE_STRIDE * sizeof(uint64_t);
  flock_once_per_device((const void*)witness_kernel, [] {
    cudaFuncSetAttribute(witness_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(WARPS_PER_BLOCK * 3 * 32 * STAGE_STRIDE * sizeof(uint64_t)));
  });
  witness_kernel<<<(unsigned)blocks, threads, smem, stream>>>(d_in, n_in, n_total, (uint64_t*)d_z,
                                                              (uint64_t*)d_a, (uint64_t*)d_b, (uint8_t*)d_stripe); flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}
