// Ligerito PCS prover kernels (crates/flock-core/src/pcs/ligerito.rs).
//
//  * round message (ligerito.rs:3725-3773): u0 = sum f0 b0, u2 = sum (f0+f1)(b0+b1)
//    over LSB pairs, fused with the preceding fold f' = f0 + r (f0 + f1)
//    (ligerito.rs:5517-5566, partial_eval_lsb :1673-1691);
//  * OOD introduction with b_new = eq(z) evaluated on the fly from split
//    tables, returning the message and h = sum f eq (ligerito.rs:5684-5702),
//    and its glue b += beta eq(z);
//  * induced basis (ligerito.rs:1989-2160): basis[j] = sum_i alpha_i Xhat_j(q_i)
//    with Xhat_j = prod_{k in bits(j)} What_k: the transpose of the code's
//    transform applied to the weights alpha_i at the opened positions;
//  * glue b += beta * basis, row and tree-node gathers for openings.
#include "flock_internal.h"
#include "gf128.cuh"
#include "bit_outer.cuh"
#include "gf_tab.cuh"

namespace {

constexpr int LG_THREADS = 256;

__device__ __forceinline__ void block_reduce_write(gf256 a, gf256 b, gf256 c, gf128* out) {
  __shared__ gf256 red[3][LG_THREADS / 32];
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int k = 0; k < 4; k++) {
      a.r[k] ^= __shfl_xor_sync(0xffffffffu, a.r[k], off);
      b.r[k] ^= __shfl_xor_sync(0xffffffffu, b.r[k], off);
      c.r[k] ^= __shfl_xor_sync(0xffffffffu, c.r[k], off);
    }
  int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { red[0][w] = a; red[1][w] = b; red[2][w] = c; }
  __syncthreads();
  if (threadIdx.x == 0) {
    gf256 s0 = {{0, 0, 0, 0}}, s1 = s0, s2 = s0;
    for (int k = 0; k < LG_THREADS / 32; k++) { gf256_acc(s0, red[0][k]); gf256_acc(s1, red[1][k]); gf256_acc(s2, red[2][k]); }
    out[3 * blockIdx.x] = gf256_reduce(s0);
    out[3 * blockIdx.x + 1] = gf256_reduce(s1);
    out[3 * blockIdx.x + 2] = gf256_reduce(s2);
  }
}

// FOLD: in has 2 * n_out elements, bound at r into out (n_out elements); the
// message u0 = sum f0 b0, u2 = sum (f0 + f1)(b0 + b1) over the n_out-element
// state's pairs. Partials: (u0, u2, 0) per block. n_out / 2 a multiple of
// bo::TILE.
//
// The two sums run on the tensor cores (bit_outer.cuh): warps 0..7 take tiles of
// 128 pairs of f, warps 8..15 the same tiles of b (bind through r's byte tables,
// gf_tab.cuh, write, and expand the values' bits into the tile's slot), and
// one thread of a further warp issues the MMAs in tile order. Four slots are
// shared by the eight tiles in work. Bound by the shared-memory data path: 1 KB
// of table lookups and 512 bytes of operands, written and read, per pair. With both
// products as carry-less ones in the folding threads 580 us for 2^23 pairs (ALU
// 58%, issue 47%), so 391 us (the data path 76% busy); without a fold 19 us and
// 14 us for 2^18 pairs, 357 us for 2^24 (0.44 of the measured HBM rate: a tile's
// MMAs and their commit, about 500 clocks, bound it). (One lane a pair, its four
// values 64 bytes apart from the next lane's: 552 us, the uncoalesced loads taking
// a third of the data path; loads without the four steps ahead: 451 us.)
constexpr int LM_PRODUCERS = 512, LM_THREADS = LM_PRODUCERS + 32;
template <bool FOLD>
constexpr int kLmSlots = FOLD ? 4 : 6;
template <bool FOLD>
constexpr size_t kLmSmem = (FOLD ? (size_t)GF_TAB_ENTRIES * 16 : 0) + (size_t)kLmSlots<FOLD> * bo::SLOT;
static_assert(kLmSmem<true> <= 232448 && kLmSmem<false> <= 232448, "fold shared memory above the 227 KB per-block limit");

template <bool FOLD>
__global__ void __launch_bounds__(LM_THREADS, 1)
lig_fold_msg_kernel(const gf128* __restrict__ f, const gf128* __restrict__ b, size_t n_tiles, const gf128 r,
                    gf128* __restrict__ fo, gf128* __restrict__ bo_out, gf128* __restrict__ partials,
                    const FlockKernelWait kw) {
  constexpr int LM_SLOTS = kLmSlots<FOLD>, LM_AHEAD = FOLD ? 4 : 8;
  extern __shared__ __align__(128) uint8_t lm_smem[];
  // done[tau mod 8]: the MMAs of tile tau of the CTA's sequence. A tile's warps
  // come back to the same one of them every eight tiles, so nobody skips a phase
  // (a wait tells a phase from its neighbours only).
  __shared__ uint64_t full[LM_SLOTS], done[8], all_done;
  __shared__ uint32_t tmem_slot, poly[2][4][5];
  uint8_t* slots = lm_smem;
  uint4* rtab = reinterpret_cast<uint4*>(lm_smem + (size_t)kLmSlots<FOLD> * bo::SLOT);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const size_t t0 = n_tiles * blockIdx.x / gridDim.x, t1 = n_tiles * (blockIdx.x + 1) / gridDim.x;
  const int n = (int)(t1 - t0);  // at least one: gridDim.x <= n_tiles
  if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
  if (t == 0) {
    for (int k = 0; k < LM_SLOTS; k++) tc::mbar_init(&full[k], 2);
    for (int k = 0; k < 8; k++) tc::mbar_init(&done[k], 1);
    tc::mbar_init(&all_done, 1);
    tc::mbar_fence_init();
  }
  if constexpr (FOLD) {
    for (int it = t; it < 256; it += LM_THREADS) gf_tab_row_direct(r, rtab, it);
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  // columns 0..127, 128..255: the two sums' counts; 256..287: the scales, all one
  const uint32_t tmem = tmem_slot, sf = tmem + 256;
  if (warp < 4) tc::tmem_fill32(sf + ((uint32_t)(32 * warp) << 16), 0x7f7f7f7fu);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  bool ok = kw.limit != 0;
  if (t < LM_PRODUCERS) {
    const bool is_b = warp >= 8;
    const gf128* in = is_b ? b : f;
    gf128* out = is_b ? bo_out : fo;
    const uint32_t rot = t & 15;
    // the loads run LM_AHEAD steps ahead, into the next tile
    gf128 y0[LM_AHEAD], y1[LM_AHEAD];
    auto load = [&](int tau, int k) {
      const size_t i = (t0 + tau) * (2 * bo::TILE) + lane + 32 * k;
      if constexpr (FOLD) gf_load2(&in[2 * i], y0[k % LM_AHEAD], y1[k % LM_AHEAD]);
      else y0[k % LM_AHEAD] = gf_load(&in[i]);
    };
    if ((warp & 7) < n) {
#pragma unroll
      for (int k = 0; k < LM_AHEAD; k++) load(warp & 7, k);
    }
    for (int tau = warp & 7; tau < n && ok; tau += 8) {
      // value i & 1 of pair i / 2: i = 2 pair + (lane & 1), 32 consecutive i per k
      const size_t i0 = (t0 + tau) * (2 * bo::TILE) + lane;
      gf128 v[8];
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const size_t i = i0 + 32 * k;
        if constexpr (FOLD) {
          v[k] = gf_add(y0[k % LM_AHEAD], gf_mul_tab(rtab, gf_add(y0[k % LM_AHEAD], y1[k % LM_AHEAD]), rot));
          gf_store(&out[i], v[k]);
        } else {
          v[k] = y0[k % LM_AHEAD];
        }
        if (k + LM_AHEAD < 8) load(tau, k + LM_AHEAD);
        else if (tau + 8 < n) load(tau + 8, k + LM_AHEAD - 8);
      }
      // the odd lane takes the sum
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const gf128 o = gf_shfl_xor(v[k], 1);
        if (lane & 1) v[k] = gf_add(v[k], o);
      }
      const int slot = tau % LM_SLOTS;
      if (tau >= LM_SLOTS)
        ok = __all_sync(0xffffffffu, tc::mbar_wait(&done[(tau - LM_SLOTS) % 8], ((tau - LM_SLOTS) / 8) & 1, kw.limit));
      if (ok) bo::put_tile(v, slots + slot * bo::SLOT + (is_b ? bo::SIDE : 0), lane & 1);
      tc::fence_smem_for_mma();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&full[slot]);
    }
  } else if (lane == 0) {
    for (int tau = 0; tau < n && ok; tau++) {
      const int slot = tau % LM_SLOTS;
      ok = tc::mbar_wait(&full[slot], (tau / LM_SLOTS) & 1, kw.limit);
      if (!ok) break;
      tc::fence_after();
      bo::mma_slot(tc::smem_addr(slots + slot * bo::SLOT), tmem, sf, tau == 0);
      tc::mma_commit(&done[tau % 8]);
    }
    tc::mma_commit(&all_done);
  }
  __syncwarp();  // the issuing warp's other lanes stay out of its way: a lane's wait holds up the whole warp
  ok = tc::mbar_wait(&all_done, 0, kw.limit) && ok;
  if (!ok) kw.gave_up();
  __syncwarp();
  tc::fence_after();
  if (warp < 8) bo::read_quadrant(tmem + 128 * (warp >> 2), poly[warp >> 2][warp & 3]);
  tc::fence_before();
  __syncthreads();
  if (t < 2) partials[3 * blockIdx.x + t] = bo::combine(poly[t]);
  if (t == 2) partials[3 * blockIdx.x + 2] = gf_zero();
  if (warp == 0) {
    tc::mbar_wait(&all_done, 0, tc::kDrainClocks);  // committed by now, whatever gave up
    __syncwarp();
    tc::tmem_free(tmem, 512);
  }
}

// The same for small states (at most LG_SMALL_PAIRS pairs), bound by a
// thread's chain: two lanes a pair (gf_round_small). One pair: 5.2 us (one
// thread a pair, its products unrolled: 9.3 us); 2^17 pairs: 23.4 us, beyond
// which lig_fold_msg_kernel wins (2^18 pairs: 21.8 us).
constexpr size_t LG_SMALL_PAIRS = (size_t)1 << 17;
constexpr int LGS_MAX_THREADS = 256;
__global__ void __launch_bounds__(LGS_MAX_THREADS)
lig_fold_msg_small_kernel(const gf128* __restrict__ f, const gf128* __restrict__ b, size_t pairs, int fold,
                          const gf128 r, gf128* __restrict__ fo, gf128* __restrict__ bo,
                          gf128* __restrict__ partials) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < 2 * pairs;
  gf128 f0 = gf_zero(), f1 = f0, b0 = f0, b1 = f0;
  if (act) {
    if (fold) {
      f0 = gf_load(&f[2 * i]); f1 = gf_load(&f[2 * i + 1]);
      b0 = gf_load(&b[2 * i]); b1 = gf_load(&b[2 * i + 1]);
    } else {
      f0 = gf_load(&f[i]);
      b0 = gf_load(&b[i]);
    }
  }
  const gf128 p = gf_round_small<false, 1>(f0, f1, b0, b1, fold, r, gf_zero());
  if (fold && act) {
    fo[i] = f0;
    bo[i] = b0;
  }
  if (threadIdx.x == 2) partials[3 * blockIdx.x + 2] = gf_zero();
  gf_block_sum_lanes(p, 0, partials + 3 * blockIdx.x);  // u0 from the even lanes, u2 from the odd ones
}

// Message of (f, eq(z)) and h = sum f * eq(z); eq(z)[j] = lo[j & mask] * hi[j >> lo_bits].
__global__ void __launch_bounds__(LG_THREADS, 2)
lig_intro_eq_kernel(const gf128* __restrict__ f, size_t n, const gf128* __restrict__ lo,
                    const gf128* __restrict__ hi, int lo_bits, gf128* __restrict__ partials) {
  gf256 u0 = {{0, 0, 0, 0}}, u2 = u0, h = u0;
  size_t mask = ((size_t)1 << lo_bits) - 1;
  for (size_t j = (size_t)blockIdx.x * LG_THREADS + threadIdx.x; j < n / 2; j += (size_t)gridDim.x * LG_THREADS) {
    size_t i0 = 2 * j, i1 = 2 * j + 1;
    gf128 e0 = gf_mul(lo[i0 & mask], hi[i0 >> lo_bits]);
    gf128 e1 = gf_mul(lo[i1 & mask], hi[i1 >> lo_bits]);
    gf128 f0 = f[i0], f1 = f[i1];
    gf256 p0 = gf_mul_wide(f0, e0);
    gf256_acc(u0, p0);
    gf256_acc(h, p0);
    gf256_acc(h, gf_mul_wide(f1, e1));
    gf256_acc(u2, gf_mul_wide(gf_add(f0, f1), gf_add(e0, e1)));
  }
  block_reduce_write(u0, u2, h, partials);
}

// The same for small states: two lanes a pair, one product each per step
// (eq's value, f eq, then the sums' product, of which the odd lane's counts),
// through one loop body. One pair: lig_intro_eq_kernel 8.4 us, this 5.0 us.
__global__ void __launch_bounds__(LGS_MAX_THREADS)
lig_intro_eq_small_kernel(const gf128* __restrict__ f, size_t n, const gf128* __restrict__ lo,
                          const gf128* __restrict__ hi, int lo_bits, gf128* __restrict__ partials) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  gf128 v = gf_zero(), x = v, y = v, p = v, q = v;
  if (i < n) {
    v = gf_load(&f[i]);
    x = gf_load(&lo[i & (((size_t)1 << lo_bits) - 1)]);
    y = gf_load(&hi[i >> lo_bits]);
  }
#pragma unroll 1
  for (int s = 0; s < 3; s++) {
    const gf128 m = gf_mul(x, y);
    if (s == 0) {  // m = eq(z)[i]
      x = v;
      y = m;
    } else if (s == 1) {
      p = m;
      x = gf_add(x, gf_shfl_xor(x, 1));
      y = gf_add(y, gf_shfl_xor(y, 1));
    } else {
      q = m;
    }
  }
  // even lanes: p = f0 e0; odd lanes: p = f1 e1, q = (f0 + f1)(e0 + e1)
  __shared__ gf128 red[LGS_MAX_THREADS / 32][3];
#pragma unroll
  for (int off = 16; off > 1; off >>= 1) {
    p = gf_add(p, gf_shfl_xor(p, off));
    q = gf_add(q, gf_shfl_xor(q, off));
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const gf128 both = gf_add(p, gf_shfl_xor(p, 1));
  if (lane == 0) red[w][0] = p;
  if (lane == 1) {
    red[w][1] = q;
    red[w][2] = both;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    gf128 s = red[0][threadIdx.x];
    for (int k = 1; k < (int)(blockDim.x >> 5); k++) s = gf_add(s, red[k][threadIdx.x]);
    partials[3 * blockIdx.x + threadIdx.x] = s;
  }
}

__global__ void glue_eq_kernel(gf128* __restrict__ b, size_t n, const gf128* __restrict__ lo,
                               const gf128* __restrict__ hi, int lo_bits, gf128 beta) {
  size_t mask = ((size_t)1 << lo_bits) - 1;
  for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (size_t)gridDim.x * blockDim.x)
    b[j] = gf_add(b[j], gf_mul(beta, gf_mul(lo[j & mask], hi[j >> lo_bits])));
}

__global__ void glue_kernel(gf128* __restrict__ b, const gf128* __restrict__ add, size_t n, gf128 beta) {
  for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (size_t)gridDim.x * blockDim.x)
    b[j] = gf_add(b[j], gf_mul(beta, add[j]));
}

// LO[i][j] = alpha_i prod_{k < bits, bit k of j} What_k(q_i)
// (ligerito.rs:1776-1824: s_0 = q, s_k = s^2 + s_{k-1}(v_{k-1}) s, normalized by
// 1 / s_k(v_k)). Each s_k is GF(2)-linear in its argument (a square plus a
// constant multiple of a linear map), so What_k(q) is the XOR, over the set
// bits b of the 32-bit index q, of lin[k][b] = What_k(x^b): no product. CTA
// (query i, chunk c) forms those values, then the sub-tables of the low TB_LO
// bits (scaled) and of the remaining high bits (at most TB_HI) in shared
// memory, then its 256 entries with one product each.
constexpr int TB_LO = 5, TB_HI = 7, TB_THREADS = 256;
static_assert((1 << TB_LO) <= 32 && 32 + (1 << TB_HI) <= TB_THREADS, "sub-table builders fit the CTA");
__global__ void __launch_bounds__(TB_THREADS)
query_tensor_kernel(const uint32_t* __restrict__ queries, int bits, const gf128* __restrict__ lin,
                    const gf128* __restrict__ alpha, gf128* __restrict__ LO) {
  __shared__ gf128 w[TB_LO + TB_HI], lo_t[1 << TB_LO], hi_t[1 << TB_HI];
  const int lb = bits < TB_LO ? bits : TB_LO, hb = bits - lb;
  const size_t len = (size_t)1 << bits;
  const size_t chunks = (len + TB_THREADS - 1) / TB_THREADS;
  const int i = (int)(blockIdx.x / chunks);
  const size_t c = blockIdx.x % chunks;
  const int t = threadIdx.x;
  // four lanes per coordinate, eight index bits each
  if (t < 64) {  // two whole warps
    const int k = t >> 2, b0 = (t & 3) * 8;
    gf128 acc = gf_zero();
    if (k < bits) {
      const uint32_t q = queries[i] >> b0;
      const gf128* row = lin + (size_t)k * 32 + b0;
#pragma unroll
      for (int b = 0; b < 8; b++)
        if ((q >> b) & 1) acc = gf_add(acc, row[b]);
    }
#pragma unroll
    for (int off = 1; off < 4; off <<= 1)
#pragma unroll
      for (int v = 0; v < 4; v++) acc.w[v] ^= __shfl_xor_sync(0xffffffffu, acc.w[v], off);
    if ((t & 3) == 0 && k < TB_LO + TB_HI) w[k] = acc;
  }
  __syncthreads();
  // one loop for both sub-tables: a small body (the latency of a cold kernel)
  {
    const bool is_lo = t < (1 << lb), is_hi = t >= 32 && t - 32 < (1 << hb);
    const int u = is_lo ? t : t - 32, k0 = is_lo ? 0 : lb, nb = is_lo ? lb : hb;
    if (is_lo || is_hi) {
      gf128 acc = is_lo ? alpha[i] : gf_one();
#pragma unroll 1
      for (int k = 0; k < nb; k++)
        if ((u >> k) & 1) acc = gf_mul(acc, w[k0 + k]);
      if (is_lo) lo_t[u] = acc;
      else hi_t[u] = acc;
    }
  }
  __syncthreads();
  const size_t j = c * TB_THREADS + t;
  if (j < len) LO[(size_t)i * len + j] = gf_mul(lo_t[j & ((1 << lb) - 1)], hi_t[j >> lb]);
}

// The induced basis as a transposed transform. The code's position q holds
// sum_j msg_j Xhat_j(q), so basis = E^T v for the code's encoding E (the rate
// 2^-rate replication, then the additive NTT, ntt.cu) and the vector v with
// alpha_i at q_i. The low lo_bits coordinates of j are expanded per query (the
// rows LO_i of query_tensor_kernel); over the remaining pos_bits = log_d -
// lo_bits position bits the transposed layers run from the deepest up, on LO
// rows as lanes: a butterfly u' = u + t v, v' = v + u' transposes to s = u + v,
// u = s, v = v + t s; last the replicas add up. That is
// (pos_bits - rate) 2^(log_d - 1) products instead of the nq 2^n of adding
// HI_i[j_hi] LO_i[j_lo] query by query (218 queries of 2^19 coordinates:
// 1,153 us through byte tables rebuilt per query, 141 us here; 53 queries of
// 2^10: 31 us in sliced products, 10 us here).
// A CTA owns 2^log_tl lanes and all positions in shared memory, one layer
// between two barriers. Bound by the carry-less products (ALU and multiplier
// pipes) at large n, by the chain of pos_bits - rate dependent products at
// small n. The loop body stays at IB_ILP products: the first pass through a
// larger one costs more in instruction fetches than it saves (three layers
// unrolled in registers: 25 us against 7 us at 2^9 coordinates, 138 us against
// 141 us at 2^19).
constexpr int IB_THREADS = 256;
constexpr int IB_ILP = 2;
constexpr size_t IB_MAX_SMEM = (size_t)128 << 10;

// queries: sorted, distinct. tw: the plain twiddle table of 2^log_d positions
// (its first layers do not depend on which positions a lane stands for).
__global__ void __launch_bounds__(IB_THREADS, 2)
induced_basis_kernel(const gf128* __restrict__ LO, const uint32_t* __restrict__ queries, int nq, int lo_bits,
                     int pos_bits, int rate, int log_tl, const gf128* __restrict__ tw, gf128* __restrict__ basis) {
  extern __shared__ gf128 V[];  // [position][lane]
  const uint32_t tl_mask = (1u << log_tl) - 1, lane0 = blockIdx.x << log_tl;
  for (uint32_t e = threadIdx.x; e < (1u << (pos_bits + log_tl)); e += IB_THREADS) V[e] = gf_zero();
  __syncthreads();
  // several queries may share a position block
  for (uint32_t it = threadIdx.x; it < (uint32_t)nq << log_tl; it += IB_THREADS) {
    const uint32_t i = it >> log_tl, lane = it & tl_mask;
    const gf128 v = LO[((size_t)i << lo_bits) + lane0 + lane];
    uint32_t* d = V[((queries[i] >> lo_bits) << log_tl) | lane].w;
#pragma unroll
    for (int k = 0; k < 4; k++) atomicXor(d + k, v.w[k]);
  }
  __syncthreads();
  const uint32_t items = 1u << (pos_bits - 1 + log_tl);
#pragma unroll 1
  for (int t = pos_bits - 1; t >= rate; t--) {
    const int sh = pos_bits - 1 - t;
    const gf128* twl = tw + ((1u << t) - 1);
#pragma unroll 1
    for (uint32_t it0 = threadIdx.x; it0 < items; it0 += IB_ILP * IB_THREADS) {
#pragma unroll
      for (int k = 0; k < IB_ILP; k++) {
        const uint32_t it = it0 + k * IB_THREADS;
        if (it < items) {
          const uint32_t lane = it & tl_mask, g = it >> log_tl, lo = g & ((1u << sh) - 1), hi = g >> sh;
          const uint32_t p0 = (((hi << (sh + 1)) | lo) << log_tl) | lane, p1 = p0 + (1u << (sh + log_tl));
          const gf128 v = V[p1], u = gf_add(V[p0], v);
          V[p0] = u;
          V[p1] = gf_add(v, gf_mul(u, gf_load(&twl[hi])));
        }
      }
    }
    __syncthreads();
  }
  const uint32_t out_n = 1u << (pos_bits - rate);
  for (uint32_t e = threadIdx.x; e < out_n << log_tl; e += IB_THREADS) {
    gf128 acc = V[e];
    for (uint32_t c = 1; c < (1u << rate); c++) acc = gf_add(acc, V[e + ((c * out_n) << log_tl)]);
    basis[((size_t)(e >> log_tl) << lo_bits) + lane0 + (e & tl_mask)] = acc;
  }
}

// out[j] = in[2j] + r (in[2j] + in[2j+1]): one LSB fold (ligerito.rs:1673-1691).
__global__ void fold_lsb_kernel(const gf128* __restrict__ in, size_t n_out, const __grid_constant__ gf128p r,
                                gf128* __restrict__ out) {
  for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n_out; j += (size_t)gridDim.x * blockDim.x) {
    const gf128 x0 = in[2 * j], x1 = in[2 * j + 1];
    out[j] = gf_add(x0, gf_mul_p(gf_add(x0, x1), r));
  }
}

// The opened rows, then the multiproof's nodes, in one launch. The index lists
// are read from, and the values written to, pinned host memory: no copies
// before or behind the kernel.
__global__ void gather_opening_kernel(const gf128* __restrict__ mat, const uint32_t* __restrict__ rows, int n_rows,
                                      int width, gf128* __restrict__ out_rows, const uint4* __restrict__ tree,
                                      const uint32_t* __restrict__ idx, int n_nodes, uint4* __restrict__ out_nodes) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nr = (size_t)n_rows * width;
  if (e < nr) {
    const size_t r = e / width, c = e % width;
    out_rows[e] = mat[(size_t)rows[r] * width + c];
  } else if (e - nr < 2 * (size_t)n_nodes) {
    const size_t k = e - nr;
    out_nodes[k] = tree[2 * (size_t)idx[k >> 1] + (k & 1)];
  }
}

inline gf128 to_gf(const uint64_t v[2]) {
  gf128 r;
  r.w[0] = (uint32_t)v[0]; r.w[1] = (uint32_t)(v[0] >> 32); r.w[2] = (uint32_t)v[1]; r.w[3] = (uint32_t)(v[1] >> 32);
  return r;
}
inline unsigned grid_for(size_t work, size_t threads, size_t cap) {
  size_t g = (work + threads - 1) / threads;
  if (g < 1) g = 1;
  return (unsigned)(g > cap ? cap : g);
}

}  // namespace

int flock_lig_grid(size_t n_pairs) {
  return n_pairs <= LG_SMALL_PAIRS ? gf_small_grid(n_pairs) : (int)grid_for(n_pairs, LG_THREADS, 152 * 4);
}
int flock_lig_fold_grid(size_t n_pairs) {
  return n_pairs <= LG_SMALL_PAIRS ? gf_small_grid(n_pairs) : (int)grid_for(n_pairs, bo::TILE, 152);
}

int flock_launch_lig_fold_msg(const void* f, const void* b, size_t n_out, int fold, const uint64_t r[2], void* fo,
                              void* bo_out, void* partials, int grid, const FlockKernelWait& kw, cudaStream_t st) {
  if (n_out / 2 <= LG_SMALL_PAIRS) {
    if (grid != gf_small_grid(n_out / 2)) return FLOCK_ERR_SHAPE;
    lig_fold_msg_small_kernel<<<grid, gf_small_threads(n_out / 2), 0, st>>>(
        (const gf128*)f, (const gf128*)b, n_out / 2, fold, to_gf(r), (gf128*)fo, (gf128*)bo_out, (gf128*)partials);
    flock_count_launch();
    return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
  }
  const size_t n_tiles = n_out / 2 / bo::TILE;
  if ((n_out / 2) % bo::TILE || grid < 1 || (size_t)grid > n_tiles) return FLOCK_ERR_SHAPE;
  flock_once_per_device((const void*)lig_fold_msg_kernel<true>, [] {
    cudaFuncSetAttribute(lig_fold_msg_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLmSmem<true>);
    cudaFuncSetAttribute(lig_fold_msg_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLmSmem<false>);
  });
  if (fold)
    lig_fold_msg_kernel<true><<<grid, LM_THREADS, kLmSmem<true>, st>>>(
        (const gf128*)f, (const gf128*)b, n_tiles, to_gf(r), (gf128*)fo, (gf128*)bo_out, (gf128*)partials, kw);
  else
    lig_fold_msg_kernel<false><<<grid, LM_THREADS, kLmSmem<false>, st>>>(
        (const gf128*)f, (const gf128*)b, n_tiles, to_gf(r), nullptr, nullptr, (gf128*)partials, kw);
  flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}

int flock_launch_lig_intro_eq(const void* f, size_t n, const void* lo, const void* hi, int lo_bits, void* partials,
                              int grid, cudaStream_t st) {
  if (n / 2 <= LG_SMALL_PAIRS) {
    if (grid != gf_small_grid(n / 2)) return FLOCK_ERR_SHAPE;
    lig_intro_eq_small_kernel<<<grid, gf_small_threads(n / 2), 0, st>>>(
        (const gf128*)f, n, (const gf128*)lo, (const gf128*)hi, lo_bits, (gf128*)partials);
    flock_count_launch();
    return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
  }
  lig_intro_eq_kernel<<<grid, LG_THREADS, 0, st>>>((const gf128*)f, n, (const gf128*)lo, (const gf128*)hi, lo_bits,
                                                   (gf128*)partials); flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}

int flock_launch_glue_eq(void* b, size_t n, const void* lo, const void* hi, int lo_bits, const uint64_t beta[2],
                         cudaStream_t st) {
  glue_eq_kernel<<<grid_for(n, 256, 152 * 8), 256, 0, st>>>((gf128*)b, n, (const gf128*)lo, (const gf128*)hi,
                                                             lo_bits, to_gf(beta)); flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}

int flock_launch_glue(void* b, const void* add, size_t n, const uint64_t beta[2], cudaStream_t st) {
  glue_kernel<<<grid_for(n, 256, 152 * 8), 256, 0, st>>>((gf128*)b, (const gf128*)add, n, to_gf(beta)); flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}

namespace {
// Lanes (2^lo_bits) of the induced basis over n coordinates of a code of
// 2^log_d positions: half the coordinates, more where the positions would not
// fit a CTA's shared memory otherwise (two lanes of 2^12 positions).
int induce_lo_bits(int n, int log_d) {
  int k = (n + 1) / 2;
  if (log_d - k > 10) k = log_d - 10;
  if (k > TB_LO + TB_HI) k = TB_LO + TB_HI;
  return k < n ? k : n;
}
}  // namespace

size_t flock_induce_basis_rows_bytes(int n, int log_d, int nq) { return ((size_t)nq << induce_lo_bits(n, log_d)) * 16; }

int flock_launch_induce_basis(const uint32_t* d_queries, int nq, int n, int log_d, const void* what_lin,
                              const void* alpha_w, void* LO, void* basis, cudaStream_t st) {
  const int lo_bits = induce_lo_bits(n, log_d), pos_bits = log_d - lo_bits, rate = log_d - n;
  if (nq < 1 || n < 1 || rate < 0 || log_d > 30) return FLOCK_ERR_SHAPE;
  // lanes per CTA: up to four (64-byte runs of LO and basis rows) while the
  // grid keeps two CTAs per SM and the positions fit
  int log_tl = 0;
  while (log_tl < 2 && log_tl < lo_bits && ((size_t)1 << (lo_bits - log_tl - 1)) >= 256) log_tl++;
  while (log_tl > 0 && ((size_t)16 << (pos_bits + log_tl)) > IB_MAX_SMEM) log_tl--;
  const size_t smem = (size_t)16 << (pos_bits + log_tl);
  if (smem > IB_MAX_SMEM) return FLOCK_ERR_SHAPE;
  const void* tw = flock_ntt_twiddles(log_d);
  if (!tw) return FLOCK_ERR_OOM;
  const size_t chunks = (((size_t)1 << lo_bits) + TB_THREADS - 1) / TB_THREADS;
  query_tensor_kernel<<<(unsigned)((size_t)nq * chunks), TB_THREADS, 0, st>>>(
      d_queries, lo_bits, (const gf128*)what_lin, (const gf128*)alpha_w, (gf128*)LO);
  flock_count_launch();
  flock_once_per_device((const void*)induced_basis_kernel, [] {
    cudaFuncSetAttribute(induced_basis_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)IB_MAX_SMEM);
  });
  induced_basis_kernel<<<1u << (lo_bits - log_tl), IB_THREADS, smem, st>>>(
      (const gf128*)LO, d_queries, nq, lo_bits, pos_bits, rate, log_tl, (const gf128*)tw, (gf128*)basis);
  flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}

int flock_launch_gather_opening(const void* mat, const uint32_t* rows, int n_rows, int width, void* out_rows,
                                const void* tree, const uint32_t* idx, int n_nodes, void* out_nodes, cudaStream_t st) {
  const size_t n = (size_t)n_rows * width + 2 * (size_t)n_nodes;
  if (n == 0) return FLOCK_OK;
  gather_opening_kernel<<<grid_for(n, 256, 1u << 30), 256, 0, st>>>((const gf128*)mat, rows, n_rows, width,
                                                                   (gf128*)out_rows, (const uint4*)tree, idx, n_nodes,
                                                                   (uint4*)out_nodes);
  flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}

int flock_launch_fold_lsb(const void* in, size_t n_out, const uint64_t r[2], void* out, cudaStream_t st) {
  fold_lsb_kernel<<<grid_for(n_out, 256, 152 * 8), 256, 0, st>>>((const gf128*)in, n_out, gf_prepare(to_gf(r)),
                                                                 (gf128*)out);
  flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}
