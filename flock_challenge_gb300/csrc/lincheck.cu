// Lincheck kernels (crates/flock-core/src/lincheck.rs:1480-1660).
//
//  * partial fold: z_vec[i] = sum_outer z[i, outer] eq(x_outer, outer), read
//    from the byte stripe (byte (outer/8)*2^14 + i holds 8 outer bits), as a
//    bit-matrix product on the tensor cores (lincheck.rs:655-720);
//  * comb: alpha * A0^T eq_inner + B0^T eq_inner (+ beta at the constant
//    column) gathered column-wise from a CSC copy of the base matrices
//    (r1cs_setup.h);
//  (the product sumcheck rounds over (comb, z_vec), binding the top variable
//  (lincheck.rs:1242-1300), run on flock_launch_chain_round).
#include "flock_internal.h"
#include "gf128.cuh"
#include "r1cs_setup.h"
#include "tc.cuh"

namespace {

// The stripe fold as a bit-matrix product on the tensor cores (tc.cuh):
// z_vec[i], bit e = parity over the outer indices o of eq(o)[e] z[i, o], so
// M = 128 (the bits of eq), N = 2^14 columns, and the outer index is summed.
//
// A: the eq weights' bits as fp4, written once by eq_bits_kernel in the
// operand layout, a plane (32 outer indices) being [128 rows e][16 bytes]: word
// m of a row holds in its nibbles the bits 4 n + m of the plane. B: a thread
// takes four stripes of four columns, gathers each column's four bytes with
// byte permutations and masks them the same way, which expands 32 bits in five
// operations. The bits of mask m stand for 0.5, 1, 2, 0.5 in B and for 2, 1,
// 0.5, 2 in A, so every product is one or zero.
//
// A CTA owns FM_COLS columns and a range of the outer indices, in stages of
// FM_STAGE indices and FM_BUFS buffers. Sixteen warps load, expand and store B
// (words loaded FM_AHEAD stages before they are expanded) and count in on a
// barrier; one thread of a further warp has the copy engine fetch A and issues
// one MMA per 64 indices, so no expanding warp waits for another (one warp
// doing both, with a block barrier per stage, took 352 us at 2^18 outer
// indices: the tensor and shared-memory pipes at 29% and 22%). Subset-sum
// tables of eight eq weights per stripe with a lookup per byte took 422 us;
// this takes 241 us, and 28 us against 40 us at 2^14.
constexpr int FM_PRODUCERS = 512, FM_THREADS = FM_PRODUCERS + 32;
constexpr int FM_COLS = 256, FM_STAGE = 256, FM_BUFS = 4, FM_PLANES = FM_STAGE / 32, FM_AHEAD = 4;
constexpr int FM_A_PLANE = 128 * 16, FM_B_PLANE = FM_COLS * 16;
constexpr size_t FM_SMEM = (size_t)FM_BUFS * FM_PLANES * (FM_A_PLANE + FM_B_PLANE);
constexpr int FM_MAX_PARTS = 7;  // 64 column tiles x 7 = 2.95 waves of one CTA per SM
static_assert(FM_SMEM <= 232448, "fold shared memory above the 227 KB per-block limit");
static_assert(FM_PRODUCERS == 64 * FM_PLANES, "a producer takes one column word of one plane");

// One warp per plane: lane = outer index, then lane = bit row.
__global__ void __launch_bounds__(256)
eq_bits_kernel(const gf128* __restrict__ eq_lo, const gf128* __restrict__ eq_hi, int lo_bits, size_t n_planes,
               uint4* __restrict__ out) {
  const size_t plane = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (plane >= n_planes) return;
  const size_t o = plane * 32 + lane;
  const gf128 e = gf_mul(gf_load(&eq_lo[o & (((size_t)1 << lo_bits) - 1)]), gf_load(&eq_hi[o >> lo_bits]));
#pragma unroll
  for (int k = 0; k < 4; k++) {
    uint32_t row = 0;
#pragma unroll 8
    for (int b = 0; b < 32; b++) {
      const uint32_t v = __ballot_sync(0xffffffffu, (e.w[k] >> b) & 1);
      if (lane == b) row = v;
    }
    out[plane * 128 + 32 * k + lane] = make_uint4((row & 0x11111111u) << 2, row & 0x22222222u, (row >> 2) & 0x11111111u,
                                                  (row >> 1) & 0x44444444u);
  }
}

// The bytes of one column of four stripes, expanded: a row of one B plane.
__device__ __forceinline__ uint4 fm_expand(uint32_t w) {
  return make_uint4(w & 0x11111111u, w & 0x22222222u, w & 0x44444444u, (w >> 3) & 0x11111111u);
}

__global__ void __launch_bounds__(FM_THREADS, 1)
lc_fold_mma_kernel(const uint8_t* __restrict__ stripe, const uint8_t* __restrict__ eq_bits, int n_stages, int parts,
                   uint32_t* __restrict__ partials, const FlockKernelWait kw) {
  extern __shared__ __align__(128) uint8_t fm_smem[];  // A buffers, then B buffers
  __shared__ uint64_t a_full[FM_BUFS], b_full[FM_BUFS], done[FM_BUFS], all_done;
  __shared__ uint32_t tmem_slot;
  constexpr uint32_t kABytes = FM_PLANES * FM_A_PLANE, kBBytes = FM_PLANES * FM_B_PLANE;
  uint8_t* sa = fm_smem;
  uint8_t* sb = fm_smem + FM_BUFS * kABytes;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int tile = blockIdx.x % (FLOCK_K / FM_COLS), part = blockIdx.x / (FLOCK_K / FM_COLS);
  const int s_begin = (int)((long long)n_stages * part / parts), s_end = (int)((long long)n_stages * (part + 1) / parts);
  const int n = s_end - s_begin;  // at least one: parts <= n_stages
  if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
  if (t == 0) {
    for (int k = 0; k < FM_BUFS; k++) {
      tc::mbar_init(&a_full[k], 1);
      tc::mbar_init(&b_full[k], FM_PRODUCERS / 32);
      tc::mbar_init(&done[k], 1);
    }
    tc::mbar_init(&all_done, 1);
    tc::mbar_fence_init();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  // columns 0..255: the counts; 256..287: the operands' scales, all one
  const uint32_t tmem = tmem_slot, sf = tmem + 256;
  if (warp < 4) tc::tmem_fill32(sf + ((uint32_t)(32 * warp) << 16), 0x7f7f7f7fu);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  bool ok = kw.limit != 0;
  if (t < FM_PRODUCERS) {
    // column word cw (four columns) of plane g: stripes 4 g .. 4 g + 3 of a stage
    const int cw = t & 63, g = t >> 6;
    const uint8_t* src = stripe + (size_t)tile * FM_COLS + 4 * cw + (size_t)(s_begin * (FM_STAGE / 8) + 4 * g) * FLOCK_K;
    uint32_t x[FM_AHEAD][4];
    auto load = [&](int it, uint32_t (&v)[4]) {
#pragma unroll
      for (int k = 0; k < 4; k++)
        v[k] = *reinterpret_cast<const uint32_t*>(src + ((size_t)it * (FM_STAGE / 8) + k) * FLOCK_K);
    };
#pragma unroll
    for (int k = 0; k < FM_AHEAD; k++)
      if (k < n) load(k, x[k]);
    for (int it0 = 0; it0 < n; it0 += FM_AHEAD) {
#pragma unroll
      for (int k = 0; k < FM_AHEAD; k++) {
        const int it = it0 + k, b = it % FM_BUFS;
        if (it >= n) break;
        // a lane that gave up stays in step, without waiting any more: leaving, it would
        // miss its warp at the barriers below
        if (it >= FM_BUFS && ok) ok = tc::mbar_wait(&done[b], (it / FM_BUFS - 1) & 1, kw.limit);
        const uint32_t l01 = __byte_perm(x[k][0], x[k][1], 0x5140), h01 = __byte_perm(x[k][0], x[k][1], 0x7362);
        const uint32_t l23 = __byte_perm(x[k][2], x[k][3], 0x5140), h23 = __byte_perm(x[k][2], x[k][3], 0x7362);
        uint4* row = reinterpret_cast<uint4*>(sb + b * kBBytes + g * FM_B_PLANE) + cw;
        row[0] = fm_expand(__byte_perm(l01, l23, 0x5410));
        row[64] = fm_expand(__byte_perm(l01, l23, 0x7632));
        row[128] = fm_expand(__byte_perm(h01, h23, 0x5410));
        row[192] = fm_expand(__byte_perm(h01, h23, 0x7632));
        if (it + FM_AHEAD < n) load(it + FM_AHEAD, x[k]);
        tc::fence_smem_for_mma();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&b_full[b]);
      }
    }
  } else if (lane == 0) {
    auto load_a = [&](int it) {
      uint64_t* bar = &a_full[it % FM_BUFS];
      tc::mbar_expect(bar, kABytes);
      tc::bulk_load(sa + (it % FM_BUFS) * kABytes, eq_bits + (size_t)(s_begin + it) * kABytes, kABytes, bar);
    };
    int loads = 0;
    for (; loads < FM_BUFS - 1 && loads < n; loads++) load_a(loads);
    for (int it = 0; it < n && ok; it++) {
      const int b = it % FM_BUFS, j = it + FM_BUFS - 1;
      ok = tc::mbar_wait(&a_full[b], (it / FM_BUFS) & 1, kw.limit) &&
           tc::mbar_wait(&b_full[b], (it / FM_BUFS) & 1, kw.limit);
      if (!ok) break;
      tc::fence_after();
      const uint32_t a0 = tc::smem_addr(sa + b * kABytes), b0 = tc::smem_addr(sb + b * kBBytes);
#pragma unroll
      for (int q = 0; q < FM_PLANES / 2; q++)
        tc::mma_mxf4(tmem, tc::operand(a0 + 2 * q * FM_A_PLANE, FM_A_PLANE, 128),
                     tc::operand(b0 + 2 * q * FM_B_PLANE, FM_B_PLANE, 128), tc::mxf4_desc(128, FM_COLS), sf, sf + 16,
                     it > 0 || q > 0);
      tc::mma_commit(&done[b]);
      // the buffer of stage j: its last MMAs (stage j - FM_BUFS = it - 1)
      if (j < n) {
        if (j >= FM_BUFS) ok = tc::mbar_wait(&done[j % FM_BUFS], (j / FM_BUFS - 1) & 1, kw.limit);
        if (ok) load_a(loads++);
      }
    }
    tc::mma_commit(&all_done);
    // after a give-up the last copies may be on their way
    for (int j = loads < FM_BUFS ? 0 : loads - FM_BUFS; !ok && j < loads; j++)
      tc::mbar_wait(&a_full[j % FM_BUFS], (j / FM_BUFS) & 1, tc::kDrainClocks);
  }
  __syncwarp();  // the issuing warp's other lanes stay out of its way: a lane's wait holds up the whole warp
  ok = tc::mbar_wait(&all_done, 0, kw.limit) && ok;
  if (!ok) kw.gave_up();
  __syncwarp();
  tc::fence_after();
  // counts -> parities: lane = row e of quadrant warp & 3, a ballot per column
  if (t < FM_PRODUCERS) {
    const int quad = warp & 3, c_begin = (warp >> 2) * (FM_COLS / 4);
    for (int c0 = c_begin; c0 < c_begin + FM_COLS / 4; c0 += 32) {
      uint32_t r[32];
      tc::tmem_load32(tmem + ((uint32_t)(32 * quad) << 16) + c0, r);
      uint32_t keep = 0;
#pragma unroll
      for (int j = 0; j < 32; j++) {
        // counts below 2^23: the sum's low mantissa bit is the parity
        const uint32_t v = __ballot_sync(0xffffffffu, __float_as_uint(__uint_as_float(r[j]) + 8388608.0f) & 1);
        if (lane == j) keep = v;
      }
      // row r of B holds column 4 (r mod 64) + r / 64 of the tile
      const int rr = c0 + lane, col = tile * FM_COLS + 4 * (rr & 63) + (rr >> 6);
      partials[((size_t)part * FLOCK_K + col) * 4 + quad] = keep;
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::mbar_wait(&all_done, 0, tc::kDrainClocks);  // committed by now, whatever gave up
    __syncwarp();
    tc::tmem_free(tmem, 512);
  }
}

// comb[c] = alpha * sum_{r in colA(c)} eq[r] + sum_{r in colB(c)} eq[r] (+ beta at pin).
// Columns hold 0..7.4 K entries (930 + 355 on average): 21 M gathers of 16 bytes.
// Half the eq table (8192 rows, 128 KB) sits in shared memory at a time, and a
// CTA takes its columns, longest first, a warp each: random 16-byte lookups
// there take about ten clocks a warp, from L1 (the form before: a warp per
// column over the whole table in global memory, 57 us) one line each. Row indices
// are 16 bits. 48 us: the data path is 80% busy while an SM works, but each half
// waits for its longest column, a third of the time. (The next eight index loads
// in flight under the lookups: 55 us, their bounds checks cost more.)
constexpr int LCC_THREADS = 1024, LCC_ROWS = FLOCK_K / 2;
constexpr int LCC_MAX_COLS = (FLOCK_K + kLcGroups - 1) / kLcGroups + 1;
constexpr size_t LCC_SMEM = ((size_t)LCC_ROWS + 1) * 16 + (size_t)LCC_MAX_COLS * 2 * 16;
__global__ void __launch_bounds__(LCC_THREADS, 1)
lc_comb_kernel(const FlockLcMatrices M, const gf128* __restrict__ eq, gf128 alpha, gf128 beta, int pin,
               gf128* __restrict__ comb) {
  extern __shared__ gf128 lcc[];  // half the eq table, then the columns' sums (a, b)
  __shared__ int next[2];
  gf128* sums = lcc + LCC_ROWS + 1;
  const int t = threadIdx.x, lane = t & 31;
  const uint32_t g0 = M.g_ptr[blockIdx.x], n = M.g_ptr[blockIdx.x + 1] - g0;
  if (t < 2) next[t] = 0;
  if (t == 2) lcc[LCC_ROWS] = gf_zero();
  for (int half = 0; half < 2; half++) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < LCC_ROWS / LCC_THREADS; k++)
      lcc[k * LCC_THREADS + t] = gf_load(&eq[half * LCC_ROWS + k * LCC_THREADS + t]);
    __syncthreads();
    for (;;) {
      uint32_t i = 0;
      if (lane == 0) i = (uint32_t)atomicAdd(&next[half], 1);
      i = __shfl_sync(0xffffffffu, i, 0);
      if (i >= n) break;
      const uint32_t c = M.order[g0 + i];
#pragma unroll
      for (int m = 0; m < 2; m++) {
        const uint32_t *ptr = m ? M.b_ptr : M.a_ptr, *mid = m ? M.b_mid : M.a_mid;
        const uint16_t* idx = m ? M.b_idx : M.a_idx;
        const uint32_t begin = half ? mid[c] : ptr[c], end = half ? ptr[c + 1] : mid[c];
        gf128 s = gf_zero();
        // eight index loads in flight; past the end the entry behind the table, zero
        for (uint32_t k0 = begin; k0 < end; k0 += 8 * 32) {
          uint32_t r[8];
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const uint32_t k = k0 + 32 * q + lane;
            r[q] = k < end ? idx[k] : LCC_ROWS;
          }
#pragma unroll
          for (int q = 0; q < 8; q++)
            if (k0 + 32 * q < end) s = gf_add(s, lcc[r[q]]);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) s.w[q] = __reduce_xor_sync(0xffffffffu, s.w[q]);
        if (lane == 0) sums[2 * i + m] = half ? gf_add(sums[2 * i + m], s) : s;
      }
    }
  }
  __syncthreads();
  for (uint32_t i = t; i < n; i += LCC_THREADS) {
    const int c = (int)M.order[g0 + i];
    gf128 v = gf_add(gf_mul(alpha, sums[2 * i]), sums[2 * i + 1]);
    if (c == pin) v = gf_add(v, beta);
    comb[c] = v;
  }
}

// Quirky eq table (lincheck.rs:1127-1143): out[s + 64 * j] = lag[s] * eq(x_inner_rest)[j].
// A block takes four j: their eq values by eight lanes each, multiplied up in
// three steps, then one product per entry.
constexpr int LQ_MAX_REST = 8;
__global__ void __launch_bounds__(256)
lc_quirky_eq_kernel(const gf128* __restrict__ lag, const gf128* __restrict__ x_rest, int n_rest,
                    gf128* __restrict__ out) {
  __shared__ gf128 ej[4];
  const int t = threadIdx.x, i = blockIdx.x * 256 + t;
  const gf128 l = gf_load(&lag[t & 63]);
  if (t < 32) {
    const int j = blockIdx.x * 4 + (t >> 3), k = t & 7;
    gf128 e = gf_one();
    if (k < n_rest) {
      e = gf_load(&x_rest[k]);
      if (!((j >> k) & 1)) e.w[0] ^= 1;
    }
#pragma unroll 1
    for (int off = 1; off < LQ_MAX_REST; off <<= 1) e = gf_mul(e, gf_shfl_xor(e, off));
    if (k == 0) ej[t >> 3] = e;
  }
  __syncthreads();
  if (i < (64 << n_rest)) out[i] = gf_mul(l, ej[t >> 6]);
}

inline gf128 to_gf(const uint64_t v[2]) {
  gf128 r;
  r.w[0] = (uint32_t)v[0]; r.w[1] = (uint32_t)(v[0] >> 32); r.w[2] = (uint32_t)v[1]; r.w[3] = (uint32_t)(v[1] >> 32);
  return r;
}

}  // namespace

size_t flock_lc_fold_scratch_bytes(size_t n_stripes) {
  return n_stripes / 4 * FM_A_PLANE + (size_t)FM_MAX_PARTS * FLOCK_K * 16;
}

int flock_launch_lc_fold(const void* stripe, size_t n_stripes, const void* eq_lo, const void* eq_hi, int lo_bits,
                         void* scratch, void* z_vec, const FlockKernelWait& kw, cudaStream_t st) {
  constexpr size_t kPerStage = FM_STAGE / 8;
  if (n_stripes == 0 || n_stripes % kPerStage != 0 || n_stripes > ((size_t)1 << 19)) return FLOCK_ERR_SHAPE;
  const size_t n_planes = n_stripes / 4;
  uint8_t* bits = (uint8_t*)scratch;
  void* partials = bits + n_planes * FM_A_PLANE;
  eq_bits_kernel<<<(unsigned)((n_planes + 7) / 8), 256, 0, st>>>((const gf128*)eq_lo, (const gf128*)eq_hi, lo_bits,
                                                                n_planes, (uint4*)bits);
  flock_count_launch();
  if (cudaGetLastError() != cudaSuccess) return FLOCK_ERR_CUDA;
  flock_once_per_device((const void*)lc_fold_mma_kernel, [] {
    cudaFuncSetAttribute(lc_fold_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FM_SMEM);
  });
  const int n_stages = (int)(n_stripes / kPerStage);
  const int parts = n_stages < FM_MAX_PARTS ? n_stages : FM_MAX_PARTS;
  lc_fold_mma_kernel<<<(unsigned)(FLOCK_K / FM_COLS * parts), FM_THREADS, FM_SMEM, st>>>(
      (const uint8_t*)stripe, bits, n_stages, parts, (uint32_t*)(parts > 1 ? partials : z_vec), kw);
  flock_count_launch();
  if (cudaGetLastError() != cudaSuccess) return FLOCK_ERR_CUDA;
  return parts > 1 ? flock_launch_reduce_rows(partials, parts, FLOCK_K, z_vec, st) : FLOCK_OK;
}

int flock_launch_lc_comb(const FlockLcMatrices& M, const void* eq, const uint64_t alpha[2], const uint64_t beta[2],
                         int pin, void* comb, cudaStream_t st) {
  flock_once_per_device((const void*)lc_comb_kernel, [] {
    cudaFuncSetAttribute(lc_comb_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LCC_SMEM);
  });
  lc_comb_kernel<<<kLcGroups, LCC_THREADS, LCC_SMEM, st>>>(M, (const gf128*)eq, to_gf(alpha), to_gf(beta), pin,
                                                           (gf128*)comb);
  flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}

int flock_launch_lc_quirky_eq(const void* lag, const void* x_rest, int n_rest, void* out, cudaStream_t st) {
  if (n_rest < 0 || n_rest > LQ_MAX_REST) return FLOCK_ERR_SHAPE;
  int n = 64 << n_rest;
  lc_quirky_eq_kernel<<<(n + 255) / 256, 256, 0, st>>>((const gf128*)lag, (const gf128*)x_rest, n_rest,
                                                       (gf128*)out); flock_count_launch();
  return cudaGetLastError() == cudaSuccess ? FLOCK_OK : FLOCK_ERR_CUDA;
}

