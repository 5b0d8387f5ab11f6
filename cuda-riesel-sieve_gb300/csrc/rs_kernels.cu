// rs_kernels.cu -- the sieve's device kernels for sm_103a.
//
//   sieve_large_kernel, sieve_small_kernel
//                  segmented Eratosthenes over odd numbers: primes >= 65536
//                  once per window into an L2-resident bitmap, smaller ones
//                  per 2^15-odd segment in shared memory, then compaction; the
//                  primes of a p-window go straight into HBM (in ascending order
//                  by segment_scan_kernel and segment_emit_kernel).  Replaces the
//                  host prime generator generateGPUPrimes
//                  (kernel_v0.24.6.cu:1838-1987), but is complete (every
//                  composite removed) where the reference leaves composites
//                  above smallP_max^2.
//   setup_kernel   one thread per prime: Montgomery constants, B = b^Q, the
//                  quadratic-character filter per (k, n mod Q) row
//                  (kernel_v0.24.6.cu:461-521), the per-row giant-step start
//                  values k*b^r*B^e0 (kernel_v0.24.6.cu:454-509,525-528) and the
//                  per-lane power tables the BSGS kernels start from.  For
//                  integer rows (every k*b^r < 2^32) B^e0 moves into the lane
//                  table and a start value is the integer k*b^r itself.
//   bsgs_kernel    one prime per warp: baby steps B^j (j < m) in 64 chains of
//                  consecutive exponents into a shared-memory membership filter
//                  keyed by 64-bit fractions, then giant steps for every active
//                  row, 32 lanes per prime (kernel_v0.24.6.cu:365-620 is the
//                  per-thread, global-memory original).  Candidate hits are
//                  checked against the row bitmap on the device and appended with
//                  one atomic each.
//   bsgs_cta_kernel  the same with a CTA of 16 warps per prime and one large
//                  filter, for jobs with many k or wide n ranges; its tag matches
//                  are settled by settle_kernel.
//   bsgs_exact_kernel  the rare primes with too many suspects, with an exact
//                  (tag, j) table.
//   verify_kernel  direct k*b^n check of every hit (kernel_v0.24.6.cu:1649-1671).
#include <cstdio>
#include <type_traits>
#include <algorithm>

#include "rs_arith.cuh"
#include "rs_internal.h"

namespace rs {

// ---------------------------------------------------------------------------
// Segmented sieve of Eratosthenes over the odd numbers of [lo, hi], lo odd.
// Bit x of the window stands for lo + 2x.  Sieving primes q >= 2*kSieveOdds hit a
// 2^15-odd segment at most once or twice, so they are applied once per window
// by sieve_large_kernel (one thread per prime, atomicOr into an L2-resident
// bitmap of the whole window); sieve_small_kernel then starts each segment from
// that bitmap, crosses off the small primes in shared memory and compacts.

__global__ void __launch_bounds__(256) sieve_large_kernel(uint64_t lo, uint64_t hi, const uint32_t *__restrict__ sp,
                                                          const uint64_t *__restrict__ sp_rcp, uint32_t first,
                                                          uint32_t nsp, uint32_t *__restrict__ gbits, uint64_t nodd) {
  const uint32_t t = first + blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nsp) return;
  const uint32_t q = sp[t];
  const uint64_t qq = (uint64_t)q * q;
  if (qq > hi) return;
  const uint64_t start = qq > lo ? qq : lo;
  const uint32_t r = mod_rcp(start, q, sp_rcp[t]);
  uint64_t f = r ? start + (q - r) : start;
  if (!(f & 1)) f += q;
#pragma unroll 1
  for (uint64_t x = (f - lo) >> 1; x < nodd; x += q) atomicOr(&gbits[x >> 5], 1u << (x & 31));
}

// ORDERED: the segment's primes go back to gbits as bits and their number to
// seg_count, for the ordered compaction below.
// ODDS: odd numbers per segment; a window with few segments takes shorter ones.
template <bool ORDERED, int ODDS>
__global__ void __launch_bounds__(kSieveThreads)
sieve_small_kernel(uint64_t lo, uint64_t hi, const uint32_t *__restrict__ sp, const uint64_t *__restrict__ sp_rcp,
                   uint32_t nsmall, uint32_t *gbits, uint64_t *__restrict__ out, uint32_t *__restrict__ count,
                   uint32_t cap, uint32_t *__restrict__ seg_count) {
  __shared__ uint32_t bits[ODDS / 32];
  __shared__ uint32_t warp_tot[kSieveThreads / 32];
  __shared__ uint32_t block_base;
  const uint64_t base = lo + 2ull * (uint64_t)ODDS * blockIdx.x;  // odd
  if (base > hi) return;
  const uint64_t span = (hi - base) / 2 + 1;
  const uint32_t nodd = span < (uint64_t)ODDS ? (uint32_t)span : (uint32_t)ODDS;
  const uint64_t last = base + 2ull * (nodd - 1);
  const uint32_t tid = threadIdx.x;
  const uint32_t nwords = (nodd + 31) / 32;
  uint32_t *gseg = gbits + (size_t)blockIdx.x * (ODDS / 32);

  for (uint32_t w = tid; w < ODDS / 32; w += kSieveThreads) bits[w] = w < nwords ? gseg[w] : 0u;
  __syncthreads();

  // Smallest primes: the whole CTA strides over the multiples of one prime.
  uint32_t t = 0;
#pragma unroll 1
  for (; t < nsmall; t++) {
    const uint32_t q = sp[t];
    if (q >= 2 * kSieveThreads) break;
    const uint64_t qq = (uint64_t)q * q;
    if (qq > last) break;
    const uint64_t start = qq > base ? qq : base;
    const uint32_t r = mod_rcp(start, q, sp_rcp[t]);
    uint64_t f = r ? start + (q - r) : start;
    if (!(f & 1)) f += q;
    for (uint64_t x = ((f - base) >> 1) + (uint64_t)tid * q; x < nodd; x += (uint64_t)kSieveThreads * q)
      atomicOr(&bits[x >> 5], 1u << (x & 31));
  }
  // Other small primes: one prime per thread.
#pragma unroll 1
  for (uint32_t u = t + tid; u < nsmall; u += kSieveThreads) {
    const uint32_t q = sp[u];
    const uint64_t qq = (uint64_t)q * q;
    if (qq > last) break;  // sp ascending
    const uint64_t start = qq > base ? qq : base;
    const uint32_t r = mod_rcp(start, q, sp_rcp[u]);
    uint64_t f = r ? start + (q - r) : start;
    if (!(f & 1)) f += q;
    for (uint64_t x = (f - base) >> 1; x < nodd; x += q) atomicOr(&bits[x >> 5], 1u << (x & 31));
  }
  __syncthreads();

  // Compaction: each thread owns a contiguous run of words.
  constexpr uint32_t WPT = ODDS / 32 / kSieveThreads;
  uint32_t mine = 0;
  uint32_t wv[WPT];
#pragma unroll
  for (uint32_t i = 0; i < WPT; i++) {
    const uint32_t w = tid * WPT + i;
    uint32_t m = 0;
    if (w < nwords) {
      m = ~bits[w];
      const uint32_t valid = nodd - w * 32;
      if (valid < 32) m &= (1u << valid) - 1u;
    }
    wv[i] = m;
    mine += __popc(m);
  }
  const uint32_t lane = tid & 31, warp = tid >> 5;
  uint32_t incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= (uint32_t)d) incl += y;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t v = lane < kSieveThreads / 32 ? warp_tot[lane] : 0;
    uint32_t s = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, s, d);
      if (lane >= (uint32_t)d) s += y;
    }
    if (lane < kSieveThreads / 32) warp_tot[lane] = s - v;  // exclusive
    if (lane == kSieveThreads / 32 - 1) {
      if (ORDERED) seg_count[blockIdx.x] = s;
      else block_base = atomicAdd(count, s);
    }
  }
  if (ORDERED) {
#pragma unroll
    for (uint32_t i = 0; i < WPT; i++) gseg[tid * WPT + i] = wv[i];
    return;
  }
  __syncthreads();
  uint32_t pos = block_base + warp_tot[warp] + incl - mine;
#pragma unroll
  for (uint32_t i = 0; i < WPT; i++) {
    uint32_t m = wv[i];
    const uint64_t wbase = base + 2ull * 32ull * (tid * WPT + i);
    while (m) {
      const int b = __ffs(m) - 1;
      m &= m - 1;
      if (pos < cap) out[pos] = wbase + 2ull * (uint32_t)b;
      pos++;
    }
  }
}

// Exclusive prefix sums of the segments' prime counts, in place; the total to *count.
__global__ void __launch_bounds__(1024) segment_scan_kernel(uint32_t *seg, uint32_t n, uint32_t *count) {
  __shared__ uint32_t warp_tot[32];
  __shared__ uint32_t carry;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (uint32_t b = 0; b < n; b += 1024) {
    const uint32_t v = b + tid < n ? seg[b + tid] : 0;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= (uint32_t)d) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      uint32_t t = warp_tot[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, t, d);
        if (lane >= (uint32_t)d) t += y;
      }
      warp_tot[lane] = t;  // inclusive
    }
    __syncthreads();
    const uint32_t base = carry + (warp ? warp_tot[warp - 1] : 0) + incl - v;
    if (b + tid < n) seg[b + tid] = base;
    __syncthreads();
    if (tid == 1023) carry += warp_tot[31];
    __syncthreads();
  }
  if (tid == 0) *count = carry;
}

// The primes of every segment's bits in ascending order, each segment from its
// prefix sum on: as 64-bit values, or (rcp given) as sieving primes, 32-bit with
// floor(2^64 / q).
__global__ void __launch_bounds__(kSieveThreads)
segment_emit_kernel(uint64_t lo, const uint32_t *__restrict__ gbits, const uint32_t *__restrict__ seg, uint32_t cap,
                    uint64_t *__restrict__ out, uint32_t *__restrict__ out32, uint64_t *__restrict__ rcp) {
  constexpr uint32_t WPT = kSieveOdds / 32 / kSieveThreads;
  __shared__ uint32_t warp_tot[kSieveThreads / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t *g = gbits + (size_t)blockIdx.x * (kSieveOdds / 32) + tid * WPT;
  uint32_t wv[WPT], mine = 0;
#pragma unroll
  for (uint32_t i = 0; i < WPT; i++) {
    wv[i] = g[i];
    mine += __popc(wv[i]);
  }
  uint32_t incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= (uint32_t)d) incl += y;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  uint32_t pos = seg[blockIdx.x] + incl - mine;
  for (uint32_t w = 0; w < warp; w++) pos += warp_tot[w];
  const uint64_t base = lo + 2ull * kSieveOdds * blockIdx.x;
#pragma unroll
  for (uint32_t i = 0; i < WPT; i++) {
    uint32_t m = wv[i];
    const uint64_t wbase = base + 64ull * (tid * WPT + i);
    while (m) {
      const uint64_t q = wbase + 2ull * (uint32_t)(__ffs(m) - 1);
      m &= m - 1;
      if (pos < cap) {
        if (rcp) {
          out32[pos] = (uint32_t)q;
          rcp[pos] = ~0ull / q;  // floor(2^64 / q) for odd q > 1
        } else {
          out[pos] = q;
        }
      }
      pos++;
    }
  }
}

uint64_t sieve_bitmap_words(uint64_t lo, uint64_t hi) {
  const uint64_t nodd = (hi - lo) / 2 + 1;
  const uint64_t segs = (nodd + kSieveOdds - 1) / kSieveOdds;
  return segs * (kSieveOdds / 32);
}
uint32_t sieve_segments(uint64_t lo, uint64_t hi) { return (uint32_t)(sieve_bitmap_words(lo, hi) / (kSieveOdds / 32)); }

cudaError_t launch_sieve(uint64_t lo, uint64_t hi, const uint32_t *sp, const uint64_t *sp_rcp, uint32_t nsp,
                         uint32_t nsmall, uint32_t *gbits, uint64_t *out, uint32_t *count, uint32_t cap,
                         cudaStream_t st, uint32_t *seg) {
  const uint64_t nodd = (hi - lo) / 2 + 1;
  const uint32_t blocks = sieve_segments(lo, hi);
  cudaError_t e = cudaMemsetAsync(gbits, 0, sieve_bitmap_words(lo, hi) * 4, st);
  if (e != cudaSuccess) return e;
  if (nsp > nsmall) {
    const uint32_t nl = nsp - nsmall;
    sieve_large_kernel<<<(nl + 255) / 256, 256, 0, st>>>(lo, hi, sp, sp_rcp, nsmall, nsp, gbits, nodd);
  }
  if (!seg) {
    // While the blocks of segments a quarter as long are two an SM at most, a
    // window's time is one block's, and such segments are faster: both passes take 61
    // -> 56 us at 1e13 for a window of 1e5, 80 -> 69 for one of 4e6 (61 segments), 82 ->
    // 81 at 92 segments.  With more of them each block's walk over the small primes
    // counts: 83 -> 92 us at 122 segments, 105 -> 155 at 290.
    constexpr int kShort = kSieveOdds / 4;
    constexpr uint32_t kShortMax = 2 * kSms / 4;
    if (blocks <= kShortMax)
      sieve_small_kernel<false, kShort><<<(unsigned)((nodd + kShort - 1) / kShort), kSieveThreads, 0, st>>>(
          lo, hi, sp, sp_rcp, nsmall, gbits, out, count, cap, nullptr);
    else
      sieve_small_kernel<false, kSieveOdds>
          <<<blocks, kSieveThreads, 0, st>>>(lo, hi, sp, sp_rcp, nsmall, gbits, out, count, cap, nullptr);
  } else {
    sieve_small_kernel<true, kSieveOdds><<<blocks, kSieveThreads, 0, st>>>(lo, hi, sp, sp_rcp, nsmall, gbits, nullptr, nullptr, 0, seg);
    segment_scan_kernel<<<1, 1024, 0, st>>>(seg, blocks, count);
  }
  return cudaGetLastError();
}

cudaError_t launch_emit(uint64_t lo, uint64_t hi, const uint32_t *gbits, const uint32_t *seg, uint32_t cap, uint64_t *out,
                        uint32_t *out32, uint64_t *rcp, cudaStream_t st) {
  segment_emit_kernel<<<sieve_segments(lo, hi), kSieveThreads, 0, st>>>(lo, gbits, seg, cap, out, out32, rcp);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Per-prime setup, one thread per prime.

__device__ __forceinline__ uint64_t &rec_el(const JobDev &J, const ChunkBufs &cb, uint32_t e, uint32_t i) {
  return cb.recs[(size_t)i * J.rec_elems + e];
}

// 16-byte store of elements e, e+1 (e even) of a record.
__device__ __forceinline__ void rec_st2(uint64_t *rec, uint32_t e, uint64_t a, uint64_t b) {
  *reinterpret_cast<uint4 *>(rec + e) = make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
}

constexpr uint32_t kSetupRegQ = 8;  // Q up to this keeps the table of b^r*B^e0 in shared memory
constexpr uint32_t kTabChunks = 8;  // 16-byte value pairs per lane per staging round
constexpr uint32_t kTabPad = 33;    // chunk slots per staging row: 32 lanes + 1, so column reads are conflict-free

// Per-warp shared memory of the setup kernel: first the staging area of the
// lane tables, then (reused) the per-thread table of b^r*B^e0 and its Shoup
// constants.
union SetupWarpSmem {
  uint4 stage[kTabChunks][kTabPad];
  uint64_t hb[kSetupRegQ][2][32];
};

// Writes 16 consecutive table values of each of the warp's 32 records, starting
// at element e0: every lane has put its values (as pairs, chunk c = values 2c,
// 2c+1) into column `lane` of the staging area; the warp then stores whole
// record runs of 128 bytes (four records per instruction) instead of 32
// scattered 16-byte pieces.
__device__ __forceinline__ void flush_table_round(const SetupWarpSmem &S, uint64_t *recs, uint32_t rec_elems,
                                                  uint32_t i0, uint32_t n, uint32_t e0, uint32_t lane) {
  __syncwarp();
  const uint32_t c = lane & (kTabChunks - 1);
#pragma unroll
  for (uint32_t q = 0; q < 32; q += 32 / kTabChunks) {
    const uint32_t r = q + lane / kTabChunks;
    const uint4 v = S.stage[c][r];
    if (i0 + r < n) *reinterpret_cast<uint4 *>(recs + (size_t)(i0 + r) * rec_elems + e0 + 2 * c) = v;
  }
  __syncwarp();
}

// One thread per prime (a warp per 32 consecutive primes).  Lanes past the
// chunk's prime count compute on a stand-in prime and store nothing.
constexpr uint32_t kSetupKStage = 256;  // per-k records staged in shared memory (8 KB)

__global__ void __launch_bounds__(128) setup_kernel(JobDev J, ChunkBufs cb) {
  __shared__ SetupWarpSmem smem[4];
  __shared__ KInfo sk[kSetupKStage];
  // the per-k records, read by every thread of the block in the row loop
  const bool kstaged = J.nk <= kSetupKStage;
  if (kstaged)
    for (uint32_t c = threadIdx.x; c < J.nk; c += blockDim.x) sk[c] = J.kinfo[c];
  __syncthreads();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  SetupWarpSmem &S = smem[warp];
  const uint32_t i0 = blockIdx.x * blockDim.x + warp * 32;
  const uint32_t i = i0 + lane;
  const uint32_t cnt = *cb.count;
  const uint32_t n = cnt < cb.cap ? cnt : cb.cap;
  if (i0 >= n) return;  // the whole warp
  const bool live = i < n;
  const uint64_t p = live ? cb.primes[i] : 1000000007ull;
  uint64_t *rec = cb.recs + (size_t)i * J.rec_elems;
  const uint64_t b0 = p > J.base ? (uint64_t)J.base : (uint64_t)J.base % p;
  const bool pb = b0 == 0;          // p | b: no k*b^n+-1 is divisible by p (nact = 0)
  const uint64_t bmod = pb ? 1 : b0;  // keeps the arithmetic below defined
  Mont M;
  M.p = p;
  M.pinv = mont_pinv(p);
  uint64_t one, r2;
  mont_consts(p, M.pinv, one, r2);
  const uint64_t bm = montmul(bmod, r2, M);        // b in Montgomery form
  const uint64_t bq = shoup_const(bm, M.pinv);     // Shoup constant of b
  const uint64_t B = mont_pow(bm, J.Q, one, M);    // b^Q
  const uint64_t e = J.e0 >= 0 ? (uint64_t)J.e0 : (p - 1) - (uint64_t)(-J.e0) % (p - 1);
  // B^e0 times lambda.  Every baby step and giant value carries the factor
  // lambda = 2^64 mod p: the filter's keys are fractions y/p, and without it the
  // first baby steps 1, B, B^2, ... of a large p would all have keys near zero.
  const uint64_t H = montmul(mont_pow(B, e, one, M), r2, M);
  const uint64_t G = mont_pow(B, J.m, one, M);     // B^m
  const uint64_t Bc = mont_pow(B, J.chain_len, one, M);  // B^chain_len

  // Lane tables: lambda*B^(lane*chain_len) (baby chain starts) and G^(lane % tlanes + 1)
  // (giant multipliers), stepped with Shoup products by the fixed B^chain_len
  // and G, 16 values per round.
  uint64_t Bs, Gs = 0;
  {
    const uint64_t Bw = from_mont(Bc, p, M.pinv), Bq = shoup_const(Bc, M.pinv);
    uint64_t v = r2;  // lambda * B^0
#pragma unroll 1
    for (uint32_t h = 0; h < 2; h++) {
#pragma unroll 4
      for (uint32_t c = 0; c < kTabChunks; c++) {
        const uint64_t v1 = shoup_mul(v, Bw, Bq, p);
        S.stage[c][lane] = make_uint4((uint32_t)v, (uint32_t)(v >> 32), (uint32_t)v1, (uint32_t)(v1 >> 32));
        v = shoup_mul(v1, Bw, Bq, p);
      }
      flush_table_round(S, cb.recs, J.rec_elems, i0, n, J.el_tab + 16 * h, lane);
    }
    Bs = Bc;  // B^(32*chain_len)
#pragma unroll 1
    for (uint32_t q = 0; q < 5; q++) Bs = montmul(Bs, Bs, M);
    // value t of the G table is G^(t % tlanes + 1): the chain restarts at G
    // whenever t % tlanes wraps to 0 (tlanes divides 32)
    const uint64_t Gw = from_mont(G, p, M.pinv), Gq = shoup_const(G, M.pinv);
    // integer rows: the table holds Z_(t+1) = +-lambda*B^e0 * G^(t+1) instead
    uint64_t g0 = G;
    if (J.int_rows) {
      uint64_t h2 = H;
      if (J.sign > 0 && h2) h2 = p - h2;
      g0 = shoup_mul(h2, Gw, Gq, p);
    }
    uint64_t g = g0;
    uint32_t k = 0;
#pragma unroll 1
    for (uint32_t h = 0; h < 2; h++) {
#pragma unroll 1
      for (uint32_t c = 0; c < kTabChunks; c++) {
        uint64_t pair[2];
#pragma unroll
        for (uint32_t u = 0; u < 2; u++) {
          pair[u] = g;
          if (++k == J.tlanes) {
            k = 0;
            g = g0;
          } else {
            g = shoup_mul(g, Gw, Gq, p);
          }
        }
        S.stage[c][lane] =
            make_uint4((uint32_t)pair[0], (uint32_t)(pair[0] >> 32), (uint32_t)pair[1], (uint32_t)(pair[1] >> 32));
        if (h == 1 && c == kTabChunks - 1) Gs = pair[1];  // G^32 when tlanes == 32
      }
      flush_table_round(S, cb.recs, J.rec_elems, i0, n, J.el_tab + 32 + 16 * h, lane);
    }
    if (J.tlanes != 32) {
      Gs = 0;
    } else if (J.int_rows) {  // the table's last entry is Z_32: G^32 by squaring
      Gs = G;
#pragma unroll 1
      for (uint32_t q = 0; q < 5; q++) Gs = montmul(Gs, Gs, M);
    }
  }

  // HB[r] = b^r * B^e0 (Montgomery form) with the Shoup constant of HB[r] taken
  // as an integer, so the start value of row (k, r) is the single product k*HB[r]
  // (not needed for integer rows).
  // Kept per thread in shared memory (indexed by r without a select chain); the
  // staging area is free again after the last flush.
  const bool regtab = J.Q <= kSetupRegQ;
  if (regtab && !J.int_rows) {
    uint64_t h = H;
#pragma unroll 1
    for (uint32_t r = 0; r < J.Q; r++) {
      S.hb[r][0][lane] = h;
      S.hb[r][1][lane] = shoup_const(montmul(h, r2, M), M.pinv);
      h = shoup_mul(h, bmod, bq, p);
    }
  }

  // Active rows (quadratic-character filter) and their giant-step start values
  // (the integers k*b^r for integer rows), written in pairs (V) and in groups of
  // eight (row ids) as 16-byte stores.
  const int chib = legendre_k_tab(p, J.b_odd, J.b_e2, J.b_rcp, J.b_jac, J.jac_bits);
  const int chim1 = ((uint32_t)p & 3u) == 1u ? 1 : -1;  // (-1/p)
  const bool qeven = (J.Q & 1u) == 0;
  uint32_t nact = 0;
  uint64_t vprev = 0, rp0 = 0, rp1 = 0;
  uint64_t rows_on = 0;  // row_mask: the active rows as bits
  // one active row: its start value V and its row id, packed into the record
  // (integer rows: the row id only, the kernels look up k*b^r by it; row_mask:
  // one bit)
  auto emit = [&](uint64_t V, uint32_t row) {
    if (J.row_mask) {
      rows_on |= 1ull << row;
      nact++;
      return;
    }
    if (nact & 1) {
      if (live && !J.row_ids_only) rec_st2(rec, J.el_v + nact - 1, vprev, V);
    } else {
      vprev = V;
    }
    const uint64_t rbits = (uint64_t)row << (16 * (nact & 3));
    if (nact & 4) rp1 |= rbits;
    else rp0 |= rbits;
    if ((nact & 7) == 7) {
      if (live) rec_st2(rec, J.el_row + (nact >> 2) - 1, rp0, rp1);
      rp0 = rp1 = 0;
    }
    nact++;
  };
  if (regtab) {
    // Q <= 8: the rows of k are its residues present (KInfo.rmask, r ascending),
    // the active ones follow from the two characters, and V = k * HB[r]; all
    // per-k data comes from one 32-byte record (shared memory when staged).
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < J.nk; c0 += 4) {
      // the four characters first, so their table loads are in flight together;
      // kept as 2-bit fields (character + 1) so that no array goes to local memory
      uint32_t chpack = 0;
#pragma unroll
      for (uint32_t u = 0; u < 4; u++) {
        const uint32_t c = c0 + u;
        int ch = 0;
        if (c < J.nk) {
          const KInfo &ki = kstaged ? sk[c] : J.kinfo[c];
          ch = legendre_k_tab(p, ki.k_odd, ki.k_e2, ki.k_rcp, ki.k_jac, J.jac_bits);
        }
        chpack |= (uint32_t)(ch + 1) << (2 * u);
      }
#pragma unroll 1
      for (uint32_t u = 0; u < 4; u++) {
        const uint32_t c = c0 + u;
        int chik = (int)((chpack >> (2 * u)) & 3u) - 1;
        if (c >= J.nk) break;
        if (J.sign > 0) chik *= chim1;  // character of -k
        if (chik == 0) continue;        // p | k
        const KInfo ki = kstaged ? sk[c] : J.kinfo[c];
        uint32_t amask;
        if (qeven)  // even r: (k/p) = 1; odd r: (k/p)(b/p) = 1
          amask = (chik == 1 ? ki.rmask & 0x55555555u : 0u) | (chik * chib == 1 ? ki.rmask & 0xaaaaaaaau : 0u);
        else
          amask = (chib == -1 || chik == 1) ? ki.rmask : 0u;
        if (!amask) continue;
        const uint64_t kmod = p > ki.k_val ? (uint64_t)ki.k_val : (uint64_t)ki.k_val % p;
        const uint64_t kx = J.sign > 0 ? p - kmod : kmod;  // -k for k*b^n+1
#pragma unroll 1
        while (amask) {
          const uint32_t r = __ffs(amask) - 1;
          amask &= amask - 1;
          const uint32_t row = ki.row0 + __popc(ki.rmask & ((1u << r) - 1));
          emit(J.int_rows ? (J.row_ids_only || J.row_mask ? 0 : (uint64_t)__ldg(J.row_c + row))
                          : shoup_mul(kx, S.hb[r][0][lane], S.hb[r][1][lane], p),
               row);
        }
      }
    }
  } else {
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < J.nk; c0 += 4) {
      uint32_t chpack = 0;
#pragma unroll
      for (uint32_t u = 0; u < 4; u++) {
        const uint32_t c = c0 + u;
        const int ch = c < J.nk ? legendre_k_tab(p, J.k_odd[c], J.k_e2[c], J.k_rcp[c], J.k_jac[c], J.jac_bits) : 0;
        chpack |= (uint32_t)(ch + 1) << (2 * u);
      }
#pragma unroll 1
      for (uint32_t u = 0; u < 4; u++) {
        const uint32_t c = c0 + u;
        int chik = (int)((chpack >> (2 * u)) & 3u) - 1;
        if (c >= J.nk) break;
        if (J.sign > 0) chik *= chim1;  // character of -k
        if (chik == 0) continue;        // p | k
        const uint32_t r0 = J.k_row0[c], r1 = J.k_row0[c + 1];
        const uint64_t kmod = p > J.k_val[c] ? (uint64_t)J.k_val[c] : (uint64_t)J.k_val[c] % p;
        const uint64_t kx = J.sign > 0 ? p - kmod : kmod;  // -k for k*b^n+1
        uint64_t V = 0;
        uint32_t cur = 0;
        bool have = false;
#pragma unroll 1
        for (uint32_t row = r0; row < r1; row++) {
          const uint32_t r = J.row_r[row];
          const bool act = qeven ? (chik * ((r & 1u) ? chib : 1) == 1) : (chib == -1 || chik == 1);
          if (!act) continue;
          if (J.int_rows) {
            emit(J.row_ids_only || J.row_mask ? 0 : (uint64_t)__ldg(J.row_c + row), row);
            continue;
          }
          if (!have) {
            V = montmul(montmul(kx, r2, M), H, M);
            have = true;
          }
#pragma unroll 1
          for (; cur < r; cur++) V = shoup_mul(V, bmod, bq, p);
          emit(V, row);
        }
      }
    }
  }
  if (!live) return;
  if (J.row_mask) {
    rec_st2(rec, J.el_v, rows_on, 0);
  } else {
    if ((nact & 1) && !J.row_ids_only) rec[J.el_v + nact - 1] = vprev;
    if (nact & 7) rec_st2(rec, J.el_row + ((nact >> 3) << 1), rp0, rp1);
  }
  rec_st2(rec, kElP, p, M.pinv);
  rec_st2(rec, kElBm, B, Gs);
  // floor(2^64/p) is the Shoup constant of 1, whose Montgomery form is `one`
  // With (b/p) = 1 and both residues of every k present, k's two rows are both
  // active or both not, so the active rows come in adjacent (k, 0), (k, 1) pairs
  // whose start values differ by the factor b.
  const uint64_t paired = (J.pairable && chib == 1) ? 1ull << 32 : 0ull;
  rec_st2(rec, kElNact, pb ? 0 : (nact | paired), shoup_const(one, M.pinv));
  // the strides in normal form with their Shoup constants, once per prime
  rec_st2(rec, kElStw, from_mont(B, p, M.pinv), shoup_const(B, M.pinv));
  rec_st2(rec, kElGw, from_mont(Gs, p, M.pinv), shoup_const(Gs, M.pinv));
  // chain offsets: warp w of a prime's group starts its chains at B^(32w*c),
  // and a thread's second chain is 32W chains after its first
  uint64_t off = Bs;  // B^(32*c)
  if (J.cta_warps > 1) {
    uint64_t o = one;
#pragma unroll 1
    for (uint32_t w = 0; w < J.cta_warps; w++) {
      rec_st2(rec, kElWoff + 2 * w, from_mont(o, p, M.pinv), shoup_const(o, M.pinv));
      o = montmul(o, Bs, M);
    }
    off = o;  // B^(32W*c)
    rec_st2(rec, kElWoff + 2 * J.cta_warps, bmod, bq);  // b and its Shoup constant
  }
  rec_st2(rec, kElOfw, from_mont(off, p, M.pinv), shoup_const(off, M.pinv));
  if (J.by_res) rec_st2(rec, kElV, bmod, bq);
}

// Quadratic-character tables: word w of the table of odd k' holds bit t =
// ((32*w + t) / k') == +1 (Jacobi symbol), for 32*w + t < k'.  One launch
// builds the tables sel[0..nsel) of the job's list (odd parts kodd[], word
// offsets word_off[]), for k' too large for square_table_kernel and for
// selections too small for it; thread g writes word g - first[i] of table sel[i], where
// first[] are the running word counts of the selected tables.
__global__ void jacobi_table_kernel(const uint32_t *kodd, const uint32_t *word_off, const uint32_t *sel,
                                    const uint32_t *first, uint32_t nsel, uint32_t total_words, uint32_t *bits) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total_words) return;
  uint32_t lo = 0, hi = nsel;  // last selected table with first <= g
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (first[mid] <= g) lo = mid;
    else hi = mid;
  }
  const uint32_t t = sel[lo];
  const uint32_t k = kodd[t];
  const uint32_t w = g - first[lo];
  const uint32_t a0 = 32 * w;
  uint32_t out = 0;
  for (uint32_t b = 0; b < 32; b++) {
    const uint32_t a = a0 + b;
    if (a < k && jacobi32(a, k) == 1) out |= 1u << b;
  }
  bits[word_off[t] + w] = out;
}

// The same tables from squares: (a/k') is the product of (a/q) over the primes q
// that divide k' to an odd power, and the residues mod q are the squares 1, 4,
// 9, ..., two additions and a shared-memory bit apiece, against a binary-gcd loop
// of some twenty rounds an entry above.  A CTA makes the words from w0[] on of its
// table, at most kSquareSeg bits; a q with more residues than that goes through all its
// squares for each segment and keeps the ones there.
//   [residues mod q from `base` on as bits, 32 more than the segment or q (periodic)]
// XOR of their complements, 32 entries at a time, gives the table; entries with
// a common factor stay 0.
// Bound by the integer pipes (eight instructions a square): 1000 tables of k' up to
// 10^7 take 3.1 ms, by symbols 76; a table's longest CTA about 21 ps an entry.
__global__ void __launch_bounds__(1024, 1) square_table_kernel(const uint32_t *kodd, const uint32_t *word_off,
                                                               const uint32_t *sel, const uint32_t *w0s,
                                                               uint32_t *bits) {
  extern __shared__ uint32_t res[];
  __shared__ uint32_t next, primes[10];
  const uint32_t tid = threadIdx.x, NT = blockDim.x;
  const uint32_t t = sel[blockIdx.x], k = kodd[t], w0 = w0s[blockIdx.x];
  const uint32_t w1 = min(w0 + kSquareSeg / 32, (k + 31) / 32);
  uint32_t *out = bits + word_off[t];
  for (uint32_t w = w0 + tid; w < w1; w += NT) out[w] = 0xffffffffu;
  uint32_t n = k, from = 3, np = 0;  // what is left of k', whose prime factors are all >= from
  while (n > 1) {
    if (tid == 0) next = n;
    __syncthreads();
    for (uint32_t d = from + 2 * tid; d * d <= n; d += 2 * NT)
      if (n % d == 0) {
        atomicMin(&next, d);
        break;
      }
    __syncthreads();
    const uint32_t q = next;
    bool odd = false;
    do {
      n /= q;
      odd = !odd;
    } while (n % q == 0);
    from = q + 2;
    if (tid == 0) primes[np] = q;
    np++;
    if (odd) {
      const bool whole = q <= kSquareSeg;
      const uint32_t base = whole ? 0 : (uint32_t)((uint64_t)w0 * 32 % q);
      const uint32_t span = (whole ? q : 32 * (w1 - w0)) + 32;  // bits kept, at most kSquareSeg + 32
      for (uint32_t w = tid; w < (span + 31) / 32; w += NT) res[w] = 0;
      __syncthreads();
      // x = tid + 1 + i*NT: x^2 - base mod q by its differences
      const uint32_t half = (q - 1) / 2, x0 = tid + 1;
      if (x0 <= half) {
        const uint32_t d2 = (uint32_t)(2ull * NT * NT % q);
        uint32_t y = (uint32_t)(((uint64_t)x0 * x0 + q - base) % q), c = (uint32_t)((2ull * x0 + NT) * NT % q);
        for (uint32_t x = x0; x <= half; x += NT) {
          for (uint32_t e = y; e < span; e += q) atomicOr(&res[e >> 5], 1u << (e & 31));
          y += c;
          y = min(y, y - q);
          c += d2;
          c = min(c, c - q);
        }
      }
      __syncthreads();
      for (uint32_t w = w0 + tid; w < w1; w += NT) {
        const uint32_t off = whole ? 32 * w % q : 32 * (w - w0), i = off >> 5;
        out[w] ^= ~__funnelshift_r(res[i], res[i + 1], off);
      }
    }
    __syncthreads();
  }
  for (uint32_t w = w0 + tid; w < w1; w += NT) {
    uint32_t clear = 32 * w + 32 > k ? ~((1u << (k & 31)) - 1) : 0;
    for (uint32_t i = 0; i < np; i++) {
      const uint32_t q = primes[i], off = 32 * w % q;
      for (uint32_t b = off ? q - off : 0; b < 32; b += q) clear |= 1u << b;
    }
    out[w] &= ~clear;
  }
}

cudaError_t launch_jacobi_tables(const uint32_t *kodd, const uint32_t *word_off, const uint32_t *sel,
                                 const uint32_t *first, uint32_t nsel, uint32_t total_words, uint32_t *bits,
                                 cudaStream_t st) {
  if (total_words == 0 || nsel == 0) return cudaSuccess;
  jacobi_table_kernel<<<(total_words + 255) / 256, 256, 0, st>>>(kodd, word_off, sel, first, nsel, total_words,
                                                                 bits);
  return cudaGetLastError();
}

cudaError_t launch_square_tables(const uint32_t *kodd, const uint32_t *word_off, const uint32_t *sel,
                                 const uint32_t *w0, uint32_t nseg, uint32_t kmax, uint32_t *bits, cudaStream_t st) {
  if (nseg == 0) return cudaSuccess;
  const uint32_t smem = std::min(kmax, kSquareSeg) / 32 * 4 + 12;
  const cudaError_t e = cudaFuncSetAttribute((const void *)square_table_kernel,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, kSquareSeg / 32 * 4 + 12);
  if (e != cudaSuccess) return e;
  square_table_kernel<<<nseg, 1024, smem, st>>>(kodd, word_off, sel, w0, bits);
  return cudaGetLastError();
}

cudaError_t launch_setup(const JobDev &job, const ChunkBufs &cb, uint64_t odds, cudaStream_t st) {
  // (the chunk has at most `odds` primes: a narrow window need not launch a block
  // for every 128 primes its buffer could hold)
  const unsigned blocks = (unsigned)((std::min<uint64_t>(cb.cap, odds) + 127) / 128);
  setup_kernel<<<blocks, 128, 0, st>>>(job, cb);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Baby-step giant-step, one prime per warp.

// Candidate check of x = e0 + m*s - j on row `row`, then one atomic append.
__device__ __forceinline__ void record_hit(const JobDev &J, const HitBufs &hb, uint64_t p, uint32_t row,
                                           uint32_t s, uint32_t j) {
  const int64_t x = J.e0 + (int64_t)J.m * (int64_t)s - (int64_t)j;
  if (x < (int64_t)J.x_lo || x > (int64_t)J.x_hi) return;
  const uint64_t n = (uint64_t)x * J.Q + J.row_r[row];
  if (n < J.nmin || n > J.nmax) return;
  const uint32_t bit = (uint32_t)(x - J.x_lo);
  if (!J.datless) {
    const uint32_t w = J.bitmap[(size_t)row * J.words_per_row + (bit >> 5)];
    if (!((w >> (bit & 31)) & 1u)) return;
  }
  const uint32_t idx = atomicAdd(hb.raw_count, 1u);
  if (idx < hb.cap) {
    Hit h;
    h.p = p;
    h.k = J.k_val[J.row_kidx[row]];
    h.n = (uint32_t)n;
    hb.raw[idx] = h;
  }
}

// Asynchronous copy of the first `elems` (even) elements of prime i's record
// into shared memory: 16-byte cp.async chunks, one group per lane.
__device__ __forceinline__ void stage_copy(uint64_t *dst, const JobDev &J, const ChunkBufs &cb, uint32_t i,
                                           uint32_t elems, uint32_t lane) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const uint64_t *src = cb.recs + (size_t)i * J.rec_elems;
#pragma unroll 1
  for (uint32_t e = 2 * lane; e < elems; e += 64)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + 8 * e), "l"(src + e) : "memory");
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

__device__ __forceinline__ void stage_commit_empty() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void stage_wait_prev() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
__device__ __forceinline__ void stage_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Index of the n-th (from 0) set bit of a row mask (row_mask records).
__device__ __forceinline__ uint32_t nth_row(uint64_t mask, uint32_t n) {
#pragma unroll 1
  for (uint32_t t = 0; t < n; t++) mask &= mask - 1;
  return (uint32_t)(__ffsll((long long)mask) - 1);
}

struct __align__(16) Match {
  uint64_t y;     // giant value (normal form)
  uint32_t row;   // its row
  uint32_t s;     // giant index
};

// Nonzero iff some 16-bit half of x is zero: (x - 0x10001) & ~x sets bit 15 of
// the low half iff it is zero, and bit 15 of the high half iff it is zero or
// the low half borrowed (which only happens when the low half is zero).
__device__ __forceinline__ uint32_t zero_half(uint32_t x) { return (x - 0x00010001u) & ~x & 0x80008000u; }

// Fractions.  The filter's keys are fractions of residues: for a Montgomery-form
// residue u of y (u = y*2^64 mod p), u * (-p^-1) mod 2^64 = floor(y*2^64/p), the
// 64-bit fraction F64 of y/p.  Two properties make this the cheap key:
//   - it needs no reduced u: u + p gives F64 - 1;
//   - for an integer row c < 2^32 and W the F64 of the lane's multiplier Z,
//     c*W mod 2^64 = F64(c*Z mod p) - floor(c*u_Z/p), less than c < 2^32 below
//     the exact fraction: a giant step is one 32x32 high product and one
//     multiply-add, without the quotient, the remainder and its correction.
// So with F the high word of a value's exact F64, a giant step sees f in
// {F - 1, F}: baby steps must be found from both.
__device__ __forceinline__ uint64_t frac64(uint64_t u, uint64_t pinv) { return u * pinv; }

// Products for the baby chain without the final correction: from x < 2p to the
// product mod p plus 0 or p.
struct LazyShoup {  // any p < 2^63, by a full-size constant
  uint64_t w, wq, np;
  __device__ __forceinline__ uint64_t operator()(uint64_t x) const { return x * w + __umul64hi(x, wq) * np; }
};
// The short product by the integer c = b^Q: q = floor(floor(x/2^S) * K / 2^32)
// with K = floor(c * 2^(32+S) / p) < 2^32 is at most 1 + c*2^S/p + x/2^(32+S)
// below c*x/p.  The host picks S with both terms small enough (chunk_step_form),
// so that x < 2p gives a remainder below 2p again.
struct LazyShort {
  uint32_t c, K, S;
  uint64_t np;
  __device__ __forceinline__ uint64_t operator()(uint64_t x) const {
    const uint32_t q = __umulhi(__funnelshift_rc((uint32_t)x, (uint32_t)(x >> 32), S), K);
    return x * (uint64_t)c + (uint64_t)q * np;
  }
};

// Membership filter of a prime's baby steps (a Bloom filter blocked by 32-bit
// words) on the high words F of their fractions: bits sh1.. of F choose the
// word (scaled to any number of words); five bits from sh1 on and five from sh2 =
// sh1 - 5 on each rotate a fixed pattern whose bits are set in the word.  A giant
// value whose bits are all set is a suspect: a match, or one of the false
// positives (1.1e-3 at 0.56 values a word, 4e-4 at 0.3), which the scan of
// the tag list below rejects.  A giant step may see F - 1 for a value's F; that
// has another key only if the low sh2 bits of F are zero, and those values are
// stored for F - 1 too.  Against buckets of eight 16-bit tags with insert counts an insert
// is one atomic OR without a return value (no slot, no tag store, no full
// buckets), and a probe is one 4-byte load instead of a 16-byte one, which
// random addresses cost more than twice the shared-memory wavefronts.
// The patterns are the best of a random search for few false positives.
// Fewer bits a key make a step cheaper and the suspects dearer: two single bits
// measured 2.47 ns per prime against 2.38 for three on the benchmark job; two
// rotated patterns replaced both.
//
// What bounds the kernel is the integer pipes: a 32x32 high or wide product takes
// four cycles of a scheduler's multiply pipe, a low one two, an add, shift or
// logic operation two of its ALU, and the two overlap to about 75%.  On the
// benchmark job at 1e13 a baby step (short product, key, insert) takes 38 cycles
// against 36 for the reduced product and a bucket insert, and a giant step
// (key, probe) 28 against 50: 2.13 ns per prime against 2.82.
constexpr uint32_t kFilt2A = 0x22009u, kFilt2B = 0x2100005u;
// The CTA kernel probes ~64,000 values a prime: three five-bit fields (sh1, sh1 -
// 5, sh1 - 10) and rotations, 1.6e-4 false positives at 0.35 values a word.
constexpr uint32_t kFilt3A = 0x800081u, kFilt3B = 0x80005u, kFilt3C = 0x40041u;
__device__ __forceinline__ uint32_t rotl(uint32_t v, uint32_t s) { return __funnelshift_l(v, v, s); }

template <int K>
struct Filter {
  uint32_t *w;
  uint32_t mul;  // words << sh1
  uint32_t sh1;
  __device__ __forceinline__ uint32_t low() const { return sh1 - 5 * (K - 1); }  // bits below the last field
  __device__ __forceinline__ uint32_t bits(uint32_t u, uint32_t F) const {
    return K == 2 ? rotl(kFilt2A, u) | rotl(kFilt2B, F >> (sh1 - 5))
                  : rotl(kFilt3A, u) | rotl(kFilt3B, F >> (sh1 - 5)) | rotl(kFilt3C, F >> (sh1 - 10));
  }
  __device__ __forceinline__ void add(uint32_t F) const {
    const uint32_t u = F >> sh1;
    atomicOr(&w[__umulhi(u, mul)], bits(u, F));
  }
  __device__ __forceinline__ bool test(uint32_t f) const {
    const uint32_t u = f >> sh1;
    return (~w[__umulhi(u, mul)] & bits(u, f)) == 0;
  }
};

// Baby steps of one lane: two chains of `len` steps from va and vb, of which
// the first na (nb) count (all of them when FULL) and go into the filter.  The
// low 16 bits of both values' keys of step t are kept in tags[t * stride] for
// the suspects' scan.  The key is that of F64 + 1, which is exact for the
// unreduced residue and differs from the reduced one's only where the fraction's
// low word is all ones, where no giant step sees F - 1.
// A giant step sees F - 1 under another key only if F64 is less than cmax (the
// largest integer row) above a multiple of 2^(32 + low()): those are stored
// for F - 1 too.  With many low bits (EDGE false) it is enough to look at them:
// lim has them in both halves; else (EDGE) lim is the bound for F64's 32 bits
// below the last field.  The test is made for groups of N steps, since a branch
// a step costs a fifth of the loop.
template <bool FULL, bool EDGE, uint32_t N, int K, class Step>
__device__ __forceinline__ void baby_filter(const Filter<K> &F, uint32_t *tags, uint32_t stride, uint32_t lim,
                                            uint64_t va, uint64_t vb, uint32_t na, uint32_t nb, uint32_t len,
                                            uint64_t pinv, const Step &step) {
  auto group = [&](auto count, uint32_t t0) {
    constexpr uint32_t M = decltype(count)::value;
    uint32_t fa[M], fb[M], ga[M], gb[M], z = 0xffffffffu;
#pragma unroll
    for (uint32_t i = 0; i < M; i++) {
      const uint32_t t = t0 + i;
      const uint64_t xa = frac64(va, pinv) + 1, xb = frac64(vb, pinv) + 1;
      fa[i] = (uint32_t)(xa >> 32);
      fb[i] = (uint32_t)(xb >> 32);
      if (FULL || t < na) F.add(fa[i]);
      if (FULL || t < nb) F.add(fb[i]);
      const uint32_t tp = __byte_perm(fa[i], fb[i], 0x5410);
      tags[t * stride] = tp;
      if (EDGE) {
        ga[i] = __funnelshift_l((uint32_t)xa, fa[i], 32 - F.low());
        gb[i] = __funnelshift_l((uint32_t)xb, fb[i], 32 - F.low());
        z = min(z, min(ga[i], gb[i]));
      } else {
        z = __vminu2(z, tp & lim);
      }
      va = step(va);
      vb = step(vb);
    }
    if (EDGE ? z < lim : zero_half(z) != 0) {  // rare
#pragma unroll
      for (uint32_t i = 0; i < M; i++) {
        if (EDGE ? ga[i] < lim : (fa[i] & lim & 0xffffu) == 0) F.add(fa[i] - 1);
        if (EDGE ? gb[i] < lim : (fb[i] & lim & 0xffffu) == 0) F.add(fb[i] - 1);
      }
    }
  };
  uint32_t t = 0;
#pragma unroll 1
  for (; t + N <= len; t += N) group(std::integral_constant<uint32_t, N>{}, t);
#pragma unroll 1
  for (; t + 2 <= len; t += 2) group(std::integral_constant<uint32_t, 2>{}, t);
  if (t < len) group(std::integral_constant<uint32_t, 1>{}, t);
}

// A lane's giant multiplier from its table entry e (Montgomery form): the
// residue w in normal form and its Shoup constant wq = floor(w * 2^64 / p), which
// is also w's 64-bit fraction.  Integer rows: w = Z, and c*w is the giant value
// in normal form; V rows: w = G^s, and V*w its Montgomery form.
struct GiantMul {
  uint64_t wq;
  uint64_t p;
  __device__ __forceinline__ void set(uint64_t e, uint64_t mod, uint64_t pinv) {
    wq = frac64(e, pinv);
    p = mod;
  }
  __device__ __forceinline__ uint64_t w() const { return wq ? __umul64hi(wq, p) + 1 : 0; }  // from_mont(e)
};

// The start value of row slot sl: an integer k*b^r from the row ids (u16 into
// ctab), an active-row mask's list (u32) or V (u64), or V's residue.
template <int RM>
__device__ __forceinline__ uint64_t giant_start(const void *src, const uint32_t *__restrict__ ctab, uint32_t sl) {
  if constexpr (RM == kRowsIntId) return __ldg(ctab + reinterpret_cast<const uint16_t *>(src)[sl]);
  else if constexpr (RM == kRowsMask) return reinterpret_cast<const uint32_t *>(src)[sl];
  else if constexpr (RM == kRowsIntV) return (uint32_t) reinterpret_cast<const uint64_t *>(src)[sl];
  else return reinterpret_cast<const uint64_t *>(src)[sl];
}

// The exact giant value from its start value.
template <int RM>
__device__ __forceinline__ uint64_t giant_exact(uint64_t v, const GiantMul &G) {
  return RM == kRowsV ? shoup_mul(v, G.w(), G.wq, G.p) : shoup_mul32((uint32_t)v, G.w(), G.wq, G.p);
}

// The key of a giant value: F or F - 1 (see above).  w: G.w(), V rows only.
template <int RM>
__device__ __forceinline__ uint32_t giant_key(uint64_t v, const GiantMul &G, uint64_t w, uint64_t np, uint64_t pinv) {
  if constexpr (RM == kRowsV)
    return (uint32_t)(frac64(v * w + __umul64hi(v, G.wq) * np, pinv) >> 32);
  else
    return (uint32_t)v * (uint32_t)(G.wq >> 32) + __umulhi((uint32_t)v, (uint32_t)G.wq);
}

// The key F of an exact giant value y from the key f a giant step saw (F or F -
// 1).  True if the fraction's low word may be all ones, where a baby step may be
// stored under F + 1.
template <int RM>
__device__ __forceinline__ bool exact_key(uint64_t y, uint32_t f, uint64_t p, uint64_t pinv, uint32_t &F) {
  if constexpr (RM == kRowsV) {  // y in Montgomery form
    const uint64_t F64 = frac64(y, pinv);
    F = (uint32_t)(F64 >> 32);
    return (uint32_t)F64 == 0xffffffffu;
  } else {  // y in normal form: y*2^32 = F*p + r, 0 <= r < p
    if (f == 0xffffffffu && y < (p >> 1)) f = 0;  // F = 0, seen as -1
    uint64_t r = (y << 32) - (uint64_t)f * p;     // in [0, 2p)
    if (r >= p) {
      r -= p;
      f++;
    }
    F = f;
    return r + (p >> 32) + 1 >= p;
  }
}

// One giant step of the row slots of passes [g0, g1), two passes at a time:
// lane (lane_row) takes the start values of slots g*RPI + lane_row and
// (g+1)*RPI + lane_row.  Outcomes: bit i of hA (passes g0 + 2i) and hB (g0 +
// 2i + 1); at most 64 passes a call.  Slots past nact (RPI > 1) repeat a value;
// the caller drops their outcomes.
// PAIRED (RPI == 1, V rows): slots g, g+1 hold a (k, 0), (k, 1) pair, so the
// second value is the first times the integer b (the short product).
template <uint32_t RPI, int RM, bool PAIRED = false>
__device__ __forceinline__ void giant_test(const Filter<2> &F, const void *src, const uint32_t *__restrict__ ctab,
                                           uint32_t g0, uint32_t g1, uint32_t nact, uint32_t lane_row,
                                           const GiantMul &G, uint64_t np, uint64_t pinv, uint32_t &hA, uint32_t &hB,
                                           uint32_t b = 0, uint32_t rc = 0) {
  const uint64_t w = RM == kRowsV ? G.w() : 0;
  auto pass = [&](uint32_t g, uint32_t bit, auto both, uint32_t &ha, uint32_t &hb) {
    constexpr bool BOTH = decltype(both)::value;
    uint64_t va, vb = 0;
    if constexpr (RPI == 1 && RM == kRowsMask) {
      const uint2 c = *reinterpret_cast<const uint2 *>(reinterpret_cast<const uint32_t *>(src) + g);
      va = c.x;
      vb = c.y;
    } else if constexpr (RPI == 1 && RM == kRowsIntId) {
      const uint32_t rr = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const uint16_t *>(src) + g);
      va = __ldg(ctab + (rr & 0xffffu));
      if (BOTH) vb = __ldg(ctab + (rr >> 16));
    } else if constexpr (RPI == 1) {
      const uint4 v = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint64_t *>(src) + g);
      va = ((uint64_t)v.y << 32) | v.x;
      vb = ((uint64_t)v.w << 32) | v.z;
    } else {
      const uint32_t sa = g * RPI + lane_row;
      va = giant_start<RM>(src, ctab, min(sa, nact - 1));
      if (BOTH) vb = giant_start<RM>(src, ctab, min(sa + RPI, nact - 1));
    }
    uint32_t fa, fb;
    if constexpr (PAIRED && RM == kRowsV) {
      const uint64_t ya = shoup_mul(va, w, G.wq, G.p);
      fa = (uint32_t)(frac64(ya, pinv) >> 32);
      fb = (uint32_t)(frac64(mul_small(ya, b, rc, G.p), pinv) >> 32);
    } else {
      fa = giant_key<RM>(va, G, w, np, pinv);
      if (BOTH) fb = giant_key<RM>(vb, G, w, np, pinv);
    }
    if (F.test(fa)) ha |= bit;
    if (BOTH && F.test(fb)) hb |= bit;
  };
  // Two iterations of constant outcome bits at a time, then what is left.
  constexpr std::true_type two{};
  uint32_t g = g0, sh = 0;
#pragma unroll 1
  for (; g + 4 <= g1; g += 4, sh += 2) {
    uint32_t ha = 0, hb = 0;
    pass(g, 1, two, ha, hb);
    pass(g + 2, 2, two, ha, hb);
    hA |= ha << sh;
    hB |= hb << sh;
  }
  // (After 64 passes sh is 32, no shift count of a 32-bit word.  By a clamped shift in place of the
  // guard one k takes 88.1 ms for 88.6, but 131 k 69.3 for 68.3, 32 k at T = 32 21.9 ns for 20.7.)
  if (g < g1) {
    uint32_t ha = 0, hb = 0;
    if (g + 2 <= g1) {
      pass(g, 1, two, ha, hb);
      if (g + 2 < g1) pass(g + 2, 2, std::false_type{}, ha, hb);
    } else {
      pass(g, 1, std::false_type{}, ha, hb);
    }
    hA |= ha << sh;
    hB |= hb << sh;
  }
}

// The work of one prime in the warp-per-prime layout, the whole warp together:
// baby steps into the filter, giant steps tested against it, and the exact
// resolution of the suspects.  cur is the prime's staged record (header, and V
// or the row mask; nact != 0), Bl and Glm the lane's two table entries, c_lo /
// c_hi (row_mask) the lane's row constants, tags the lane's column of the tag
// list; npaired counts the primes whose rows come in pairs (kStatPaired).  Shared
// by the single-job kernel and the multi-job kernel below.
template <int TL, int RM>
__device__ __forceinline__ void bsgs_prime(const JobDev &J, const ChunkBufs &cb, const HitBufs &hb, uint32_t *fwords,
                                           uint32_t nw, uint32_t *tags, uint32_t *vbuf,
                                           const uint64_t *cur, uint32_t i, uint32_t nact, uint64_t Bl,
                                           uint64_t Glm, uint32_t lane, uint32_t c_lo, uint32_t c_hi,
                                           uint32_t &npaired) {
  constexpr uint32_t RPI = 32 / TL;  // row slots per lane-group pass
  const uint32_t lane_row = lane / TL;
  const uint32_t spl = TL == 32 ? J.steps_per_lane : 1;
  if constexpr (RM == kRowsMask) {  // V from the active-row mask
    const uint64_t am = cur[kElV];
    const uint32_t lo = (uint32_t)am, hi = (uint32_t)(am >> 32), below = (1u << lane) - 1u;
    if ((lo >> lane) & 1u) vbuf[__popc(lo & below)] = c_lo;
    if ((hi >> lane) & 1u) vbuf[__popc(lo) + __popc(hi & below)] = c_hi;
  }
  // By residue: the active rows' k (ks) and ids (rid) in one list per residue r,
  // from slot J.row_base[r] on, in any order; their numbers in vbuf[0..Q).
  uint32_t *ks = vbuf + kResMax;
  uint16_t *rid = reinterpret_cast<uint16_t *>(ks + J.row_slots);
  if constexpr (RM == kRowsRes) {
    if (lane < kResMax) vbuf[lane] = 0;
    __syncwarp();
    const uint16_t *ids = reinterpret_cast<const uint16_t *>(cur + J.el_row);
#pragma unroll 1
    for (uint32_t a = lane; a < ((nact + 31) & ~31u); a += 32) {
      const bool on = a < nact;
      const uint32_t id = on ? ids[a] : 0;
      const uint2 kr = __ldg(J.row_kr + id);
      const uint32_t r = on ? kr.y & 0xfffu : 0xffffffffu;
      const uint32_t same = __match_any_sync(0xffffffffu, r);
      const uint32_t have = on ? vbuf[r] : 0;
      __syncwarp();
      const uint32_t at = have + __popc(same & ((1u << lane) - 1u));
      if (on) {
        ks[at + (kr.y >> 12)] = kr.x;
        rid[at + (kr.y >> 12)] = (uint16_t)id;
        if ((same >> lane) == 1u) vbuf[r] = at + 1;  // the last of its residue
      }
      __syncwarp();
    }
  }
  const uint64_t p = cur[kElP], pinv = cur[kElPinv];
  // Multipliers in normal form with their Shoup constants; the values
  // they multiply stay in Montgomery form, so products stay comparable.
  const uint64_t Stw = cur[kElStw], Stq = cur[kElStq];
  const uint64_t np = 0 - p;
  Filter<2> F;
  F.w = fwords;
  F.sh1 = J.fshift;
  F.mul = nw << J.fshift;
  const uint32_t lim = 0x10001u * ((1u << F.low()) - 1u);
  // chain starts B^(lane*CL) and B^((lane+32)*CL); valid steps na, nb (j < m)
  const uint32_t CL = J.chain_len;
  const uint32_t ja0 = lane * CL, jb0 = ja0 + 32 * CL;
  const uint32_t na = J.m > ja0 ? min(CL, J.m - ja0) : 0;
  const uint32_t nb = J.m > jb0 ? min(CL, J.m - jb0) : 0;
  const uint64_t Blb = shoup_mul(Bl, cur[kElOfw], cur[kElOfq], p);
  const uint4 z4 = make_uint4(0, 0, 0, 0);
#pragma unroll 4
  for (uint32_t q = lane; q < nw / 4; q += 32) reinterpret_cast<uint4 *>(fwords)[q] = z4;
  __syncwarp();

  // Baby steps: chain A owns j = ja0 + t, chain B j = jb0 + t.
  auto baby = [&](auto step) {
    if (J.m == 64 * CL)  // every chain full (the planner's usual choice of m)
      baby_filter<true, false, 6>(F, tags, 32, lim, Bl, Blb, na, nb, CL, pinv, step);
    else
      baby_filter<false, false, 6>(F, tags, 32, lim, Bl, Blb, na, nb, CL, pinv, step);
  };
  if (cb.small_step == kStepShoup) baby(LazyShoup{Stw, Stq, np});
  else baby(LazyShort{J.bq_small, (uint32_t)(Stq >> (32 - cb.step_shift)), cb.step_shift, np});
  __syncwarp();

  // Giant steps: a lane takes row slots g*RPI + lane_row for two consecutive
  // passes g at a time, giant indices s = lane % TL + 1 + 32u.
  // the form of the start values: by residue the lists hold integers, as a mask's
  constexpr int GM = RM == kRowsRes ? kRowsMask : RM == kRowsFew ? kRowsV : RM;
  constexpr bool V = GM == kRowsV;
  uint32_t n = nact;  // the rows gone through: all active ones, or those of residue r
  uint32_t r = 0, base = 0;
  uint64_t E = Glm;  // the lane's multiplier as stored, advanced by G^32 per step u
  uint64_t Er = Glm; // ... for u = 0
  if constexpr (RM == kRowsRes) {
    for (; vbuf[r] == 0; r++) Er = shoup_mul(Er, cur[kElV], cur[kElV + 1], p);
    n = vbuf[r];
    base = __ldg(J.row_base + r);
    E = Er;
  }
  uint32_t ngi = (n + RPI - 1) / RPI;
  // the start values (or row ids): built by the warp, staged, or in the record
  const void *src_s = RM == kRowsRes    ? (const void *)(ks + base)
                      : RM == kRowsMask ? (const void *)vbuf
                                        : RM == kRowsIntId ? (const void *)(cur + J.el_row) : (const void *)(cur + kElV);
  const void *src_g = cb.recs + (size_t)i * J.rec_elems + (RM == kRowsIntId ? J.el_row : kElV);
  const bool staged = RM == kRowsRes || RM == kRowsMask || J.stage_full;
  // (k, 0), (k, 1) row pairs.  V rows form the second value by the short product
  // by b (p > 2^33, b*p < 2^63: mul_small); integer rows, whose key costs less than
  // that, and few V rows of many steps take each row by itself and are counted only.
  const bool paired = RPI == 1 && cb.pair_ok && staged && (cur[kElNact] >> 32);
  npaired += paired;
  // A lane's further steps (T > 32): advance the multiplier once and go through
  // the rows again; in blocks of at most 64 tests a lane, after which the block's
  // suspects are settled.  Few V rows (kRowsFew): advance two rows' values by G^32, in
  // unreduced form, through their steps.  A multiplier costs a product and its w,
  // as much as a row, which pays with more rows, four to a loop.
  GiantMul G;
  G.set(E, p, pinv);
  auto start = [&](uint32_t sl) {
    return staged ? giant_start<GM>(src_s, J.row_c, sl) : giant_start<GM>(src_g, J.row_c, sl);
  };
  uint32_t u = 0, at = 0, suspects = 0;  // step, the block's first pass, suspects so far
  const uint32_t per = min(spl, 32u);    // kRowsFew: steps of a row in a block (both powers of two)
  uint64_t ya = 0, yb = 0;               // ... the two rows' values
#pragma unroll 1
  while (true) {
    const uint32_t g1 = min(ngi, at + 64), u0 = u, at0 = at;
    uint32_t hA = 0, hB = 0;
    if constexpr (RM == kRowsFew) {
      const LazyShoup by_g{cur[kElGw], cur[kElGq], np};
      uint32_t sh = 0;
#pragma unroll 1
      do {
        if (u == 0) {
          const LazyShoup first{G.w(), G.wq, np};
          ya = first(start(at));
          if (at + 1 < n) yb = first(start(at + 1));
        } else {
          ya = by_g(ya);
          yb = by_g(yb);
        }
        auto steps = [&](auto both) {
          constexpr bool BOTH = decltype(both)::value;
#pragma unroll 1
          for (const uint32_t end = sh + per;;) {
            if (F.test((uint32_t)(frac64(ya, pinv) >> 32))) hA |= 1u << sh;
            if (BOTH && F.test((uint32_t)(frac64(yb, pinv) >> 32))) hB |= 1u << sh;
            if (++sh == end) break;
            ya = by_g(ya);
            if (BOTH) yb = by_g(yb);
          }
        };
        if (at + 1 < n) steps(std::true_type{});
        else steps(std::false_type{});
        u += per;
        if (u == spl) {
          u = 0;
          at += 2;
        }
      } while (sh < 32 && at < n);
    } else
    // Separate calls for staged and global V keep each load's address
    // space known to the compiler.
    if (RM == kRowsV && paired)
      giant_test<RPI, GM, RPI == 1>(F, src_s, J.row_c, at, g1, n, lane_row, G, np, pinv, hA, hB, J.base,
                                    (uint32_t)cur[kElRcp]);
    else if (staged)
      giant_test<RPI, GM>(F, src_s, J.row_c, at, g1, n, lane_row, G, np, pinv, hA, hB);
    else
      giant_test<RPI, GM>(F, src_g, J.row_c, at, g1, n, lane_row, G, np, pinv, hA, hB);
    // Suspects: every lane forms the exact value and key of its next one, then
    // the warp takes them in turn: each lane scans its own tags (its two chains,
    // 16 bits of each value's key), and a tag match is settled by walking the
    // two chains again in the exact values' form.
    uint64_t bits = ((uint64_t)hB << 32) | hA;
#pragma unroll 1
    while (uint32_t any = __ballot_sync(0xffffffffu, bits != 0)) {
      const uint32_t bit = bits ? __ffsll((long long)bits) - 1 : 0;
      uint32_t sl = (at + 2 * (bit & 31) + (bit >> 5)) * RPI + lane_row, su = 0;
      GiantMul M = G;
      if constexpr (RM == kRowsFew) {  // the multiplier of step su, by powers of G^32
        sl = at0 + 2 * ((bit & 31) / per) + (bit >> 5);
        su = u0 + (bit & 31) % per;
        uint64_t e = Glm, q = cur[kElGs];
#pragma unroll 1
        for (uint32_t x = su; x; x >>= 1) {
          if (x & 1) e = montmul(e, q, p, pinv);
          q = montmul(q, q, p, pinv);
        }
        M.set(e, p, pinv);
      }
      const bool mine = bits != 0 && sl < n;
      bits &= bits - 1;
      any = __ballot_sync(0xffffffffu, mine);
      suspects += __popc(any);
      if (suspects > J.match_cap) {  // the exact path takes the prime
        if (lane == 0) {
          const uint32_t r = atomicAdd(cb.redo_count, 1u);
          if (r < cb.cap) cb.redo[r] = i;
        }
        return;
      }
      uint64_t y = 0;
      uint32_t f = 0;
      bool edge = false;
      if (mine) {
        const uint64_t v = start(sl);
        y = giant_exact<GM>(v, M);
        edge = exact_key<GM>(y, giant_key<GM>(v, M, V ? M.w() : 0, np, pinv), p, pinv, f);
      }
      const uint32_t both = __ballot_sync(0xffffffffu, edge);  // these could be stored under F + 1 too
#pragma unroll 1
      for (uint32_t h = 0; h < 2; h++) {
#pragma unroll 1
        for (uint32_t left = h ? both : any; left; left &= left - 1) {
          const int src = __ffs(left) - 1;
          const uint32_t T = __byte_perm(__shfl_sync(0xffffffffu, f, src) + h, 0, 0x1010);
          uint32_t z = 0xffffffffu;
#pragma unroll 6
          for (uint32_t t = 0; t < CL; t++) z = __vminu2(z, tags[t * 32] ^ T);
          if (!__any_sync(0xffffffffu, zero_half(z))) continue;
          const uint64_t ys = __shfl_sync(0xffffffffu, y, src);
          const uint32_t slot = __shfl_sync(0xffffffffu, sl, src);
          const uint32_t step = RM == kRowsFew ? __shfl_sync(0xffffffffu, su, src) : u;
          uint64_t va = V ? Bl : from_mont(Bl, p, pinv);
          uint64_t vb = V ? Blb : from_mont(Blb, p, pinv);
#pragma unroll 1
          for (uint32_t t = 0; t < CL; t++) {
            const bool ma = va == ys && t < na, mb = vb == ys && t < nb;
            if (ma || mb) {
              const uint32_t s = ((uint32_t)src & (TL - 1)) + 1 + 32 * step;
              uint32_t row;
              if constexpr (RM == kRowsMask) {
                row = nth_row(cur[kElV], slot);
              } else if constexpr (RM == kRowsRes) {
                row = rid[base + slot];
              } else {
                const uint64_t pk = rec_el(J, cb, J.el_row + (slot >> 2), i);
                row = (uint32_t)(pk >> (16 * (slot & 3))) & 0xffffu;
              }
              if (ma) record_hit(J, hb, p, row, s, ja0 + t);
              if (mb) record_hit(J, hb, p, row, s, jb0 + t);
            }
            va = shoup_mul(va, Stw, Stq, p);
            vb = shoup_mul(vb, Stw, Stq, p);
          }
        }
      }
    }
    if constexpr (RM == kRowsFew) {
      if (at < n) continue;
      return;
    }
    at = g1;
    if (at < ngi) continue;
    at = 0;
    if (++u < spl) {
      E = shoup_mul(E, cur[kElGw], cur[kElGq], p);
    } else if constexpr (RM == kRowsRes) {  // the next residue that has rows
      u = 0;
      do {
        if (++r >= J.Q) return;
        Er = shoup_mul(Er, cur[kElV], cur[kElV + 1], p);
      } while (vbuf[r] == 0);
      n = vbuf[r];
      ngi = (n + RPI - 1) / RPI;
      base = __ldg(J.row_base + r);
      src_s = ks + base;
      E = Er;
    } else {
      break;
    }
    G.set(E, p, pinv);
  }
}

// Per-warp shared memory of the fast kernel:
//   [filter, fwords x 4 B][tags, chain_len x 32 x 4 B][2 stages x stage_elems x 8 B]
//   ([kMaskRows V x 4 B], row_mask; [kResMax counts x 4 B][k and ids of the rows,
//   row_slots x 6 B], by_res)
// The stages hold a record's header and V (double-buffered with cp.async); each
// lane's B^lane and G^(lane+1) entries are loaded into registers one prime ahead.
// With row_mask the stage holds the header and the active-row mask, and the
// warp writes V (the integers k*b^r of the active rows, in row order) into its
// own buffer from the constants of rows lane and lane + 32 that each lane keeps
// in registers.
//
// Each lane runs two independent chains in both phases (baby steps j = lane*c + t
// and j = (lane + 32)*c + t, c the chain length; giant steps on two row slots
// at a time), so that dependent products overlap.
// TL = giant steps handled side by side per row (min(T, 32)); RM = the form
// of the giant-step start values (kRowsV to kRowsFew).
template <int TL, int RM>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, 4)
bsgs_kernel(JobDev J, ChunkBufs cb, HitBufs hb) {
  extern __shared__ uint4 smem4[];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t *base = reinterpret_cast<uint8_t *>(smem4) + (size_t)warp * J.warp_smem;
  uint32_t *fwords = reinterpret_cast<uint32_t *>(base);
  uint32_t *tags = fwords + J.fwords + lane;
  uint64_t *stage0 = reinterpret_cast<uint64_t *>(fwords + J.fwords + 32 * J.chain_len);
  uint32_t *vbuf = reinterpret_cast<uint32_t *>(stage0 + 2 * J.stage_elems);  // row_mask: V of the current prime
  const uint32_t total = *cb.count;
  const uint32_t n = total < cb.cap ? total : cb.cap;
  const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
  const uint32_t first = blockIdx.x * kWarpsPerBlock + warp;
  const uint64_t *ltab = cb.recs + J.el_tab + lane;  // this lane's B^lane; G^(lane+1) 32 further

  uint64_t nBl = 0, nGl = 0;
  uint32_t npaired = 0;  // primes of this warp whose rows come in pairs
  uint32_t c_lo = 0, c_hi = 0;  // row_mask: k*b^r of rows lane and lane + 32
  if constexpr (RM == kRowsMask) {
    c_lo = lane < J.nrows ? __ldg(J.row_c + lane) : 0u;
    c_hi = lane + 32 < J.nrows ? __ldg(J.row_c + lane + 32) : 0u;
  }
  if (first < n) {
    stage_copy(stage0, J, cb, first, J.stage_elems, lane);
    nBl = __ldg(ltab + (size_t)first * J.rec_elems);
    nGl = __ldg(ltab + (size_t)first * J.rec_elems + 32);
  } else {
    stage_commit_empty();
  }

#pragma unroll 1
  for (uint32_t it = 0;; it++) {
    const uint32_t i = first + it * nwarps;
    if (i >= n) break;
    const uint64_t *cur = stage0 + (it & 1) * J.stage_elems;
    uint64_t *nxt = stage0 + ((it + 1) & 1) * J.stage_elems;
    const uint64_t Bl = nBl, Glm = nGl;
    if (i + nwarps < n) {
      stage_copy(nxt, J, cb, i + nwarps, J.stage_elems, lane);
      nBl = __ldg(ltab + (size_t)(i + nwarps) * J.rec_elems);
      nGl = __ldg(ltab + (size_t)(i + nwarps) * J.rec_elems + 32);
    } else {
      stage_commit_empty();
    }
    stage_wait_prev();
    __syncwarp();
    const uint32_t nact = (uint32_t)cur[kElNact];
    if (nact != 0)
      bsgs_prime<TL, RM>(J, cb, hb, fwords, J.fwords, tags, vbuf, cur, i, nact, Bl, Glm, lane, c_lo, c_hi, npaired);
    __syncwarp();
  }
  stage_wait_all();
  if (lane == 0 && npaired) atomicAdd(&hb.stat[kStatPaired], (unsigned long long)npaired);
}

// The warp-per-prime BSGS over many jobs in one persistent launch (the batched
// form): the primes of every item's chunk form one index space, and each warp
// walks it with the grid stride, so the work of small and large jobs spreads
// over the whole GPU in one launch instead of one launch per job.  Every item
// has its own constants (JobDev, read from global memory), records, hit buffers
// and baby-step product; all items share the template's giant lanes TL and
// start-value form RM.  Per-warp shared memory, in fixed places whatever the
// item:
//   [2 stages x stage_max x 8 B]([kMaskRows V x 4 B], RM = kRowsMask)
//   ([kResMax counts x 4 B][row_slots_max x 6 B], RM = kRowsRes)[the item's filter, fwords x 4 B, and tags, chain_len x 32 x 4 B]
// The record of the warp's next prime (possibly another item's) is staged by
// cp.async while the current one runs, as in bsgs_kernel.
template <int TL, int RM>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, kWarpCtas)
bsgs_batch_kernel(const BatchItem *__restrict__ items, uint32_t nitems, uint32_t warp_bytes, uint32_t stage_max,
                  uint32_t row_slots_max) {
  extern __shared__ uint4 smem4[];
  __shared__ uint32_t start[kBatchMaxItems + 1];  // prefix sums of the items' prime counts
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the items' prime counts, loaded in parallel, then their prefix sums
  for (uint32_t k = threadIdx.x; k < nitems; k += blockDim.x) {
    const uint32_t c = *items[k].cb.count, cap = items[k].cb.cap;
    start[k + 1] = c < cap ? c : cap;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    start[0] = 0;
    for (uint32_t k = 0; k < nitems; k++) start[k + 1] += start[k];
  }
  __syncthreads();
  const uint32_t total = start[nitems];
  uint8_t *base = reinterpret_cast<uint8_t *>(smem4) + (size_t)warp * warp_bytes;
  uint64_t *stage0 = reinterpret_cast<uint64_t *>(base);
  uint32_t *vbuf = reinterpret_cast<uint32_t *>(stage0 + 2 * stage_max);
  uint32_t *fwords = vbuf + (RM == kRowsMask ? kMaskRows : RM == kRowsRes ? kResMax + row_slots_max * 6 / 4 : 0);
  const uint32_t nwarps = gridDim.x * kWarpsPerBlock;
  const uint32_t first = blockIdx.x * kWarpsPerBlock + warp;
  // the item of global index g, from the item of an earlier (smaller) index
  auto locate = [&](uint32_t g, uint32_t k) {
    while (k + 1 < nitems && g >= start[k + 1]) k++;
    return k;
  };

  uint64_t nBl = 0, nGl = 0;
  uint32_t nk = 0;               // item of the staged next prime
  uint32_t ck = 0xffffffffu;     // item whose row constants the lanes hold
  uint32_t c_lo = 0, c_hi = 0;
  uint32_t npaired = 0;          // paired primes of item ck not yet added to its counter
  auto prefetch = [&](uint32_t g, uint64_t *dst) {
    nk = locate(g, nk);
    const BatchItem &X = items[nk];
    const uint32_t i = g - start[nk];
    stage_copy(dst, X.J, X.cb, i, X.J.stage_elems, lane);
    const uint64_t *lt = X.cb.recs + (size_t)i * X.J.rec_elems + X.J.el_tab + lane;
    nBl = __ldg(lt);
    nGl = __ldg(lt + 32);
  };
  if (first < total) prefetch(first, stage0);
  else stage_commit_empty();

#pragma unroll 1
  for (uint32_t it = 0;; it++) {
    const uint32_t g = first + it * nwarps;
    if (g >= total) break;
    const uint32_t k = nk;
    const uint32_t i = g - start[k];
    const uint64_t *cur = stage0 + (it & 1) * stage_max;
    uint64_t *nxt = stage0 + ((it + 1) & 1) * stage_max;
    const uint64_t Bl = nBl, Glm = nGl;
    if (g + nwarps < total) prefetch(g + nwarps, nxt);
    else stage_commit_empty();
    const BatchItem &X = items[k];
    if (k != ck) {
      if (lane == 0 && npaired) atomicAdd(&items[ck].hb.stat[kStatPaired], (unsigned long long)npaired);
      npaired = 0;
      ck = k;
      if constexpr (RM == kRowsMask) {
        c_lo = lane < X.J.nrows ? __ldg(X.J.row_c + lane) : 0u;
        c_hi = lane + 32 < X.J.nrows ? __ldg(X.J.row_c + lane + 32) : 0u;
      }
    }
    stage_wait_prev();
    __syncwarp();
    const uint32_t nact = (uint32_t)cur[kElNact];
    if (nact != 0)
      bsgs_prime<TL, RM>(X.J, X.cb, X.hb, fwords, X.J.fwords, fwords + X.J.fwords + lane, vbuf, cur, i, nact, Bl,
                         Glm, lane, c_lo, c_hi, npaired);
    __syncwarp();
  }
  stage_wait_all();
  if (lane == 0 && npaired && ck < nitems) atomicAdd(&items[ck].hb.stat[kStatPaired], (unsigned long long)npaired);
}

typedef void (*BatchFn)(const BatchItem *, uint32_t, uint32_t, uint32_t, uint32_t);

template <int RM>
static BatchFn batch_fn_t(uint32_t tlanes) {
  switch (tlanes) {
    case 1: return bsgs_batch_kernel<1, RM>;
    case 2: return bsgs_batch_kernel<2, RM>;
    case 4: return bsgs_batch_kernel<4, RM>;
    case 8: return bsgs_batch_kernel<8, RM>;
    case 16: return bsgs_batch_kernel<16, RM>;
    default: return bsgs_batch_kernel<32, RM>;
  }
}

typedef void (*BsgsFn)(JobDev, ChunkBufs, HitBufs);

template <int RM>
static BsgsFn bsgs_fn_t(uint32_t tlanes) {
  switch (tlanes) {
    case 1: return bsgs_kernel<1, RM>;
    case 2: return bsgs_kernel<2, RM>;
    case 4: return bsgs_kernel<4, RM>;
    case 8: return bsgs_kernel<8, RM>;
    case 16: return bsgs_kernel<16, RM>;
    default: return bsgs_kernel<32, RM>;
  }
}

static BsgsFn bsgs_fn(const JobDev &job) {
  switch (row_mode(job)) {
    case kRowsFew: return bsgs_kernel<32, kRowsFew>;
    case kRowsRes: return bsgs_fn_t<kRowsRes>(job.tlanes);
    case kRowsMask: return bsgs_fn_t<kRowsMask>(job.tlanes);
    case kRowsIntId: return bsgs_fn_t<kRowsIntId>(job.tlanes);
    case kRowsIntV: return bsgs_fn_t<kRowsIntV>(job.tlanes);
    default: return bsgs_fn_t<kRowsV>(job.tlanes);
  }
}


int bsgs_smem_bytes(const JobDev &job) {
  return job.cta_warps > 1 ? (int)job.warp_smem : kWarpsPerBlock * (int)job.warp_smem;
}

// Giant steps of the CTA kernel for one residue r: warp w of W takes groups w, w +
// W, ... of four of the n active rows (ks: their k, or rid and the job's row_k),
// multiplied by the lane's Z*b^r for one or two steps u (G0, G1).  Suspects are
// listed as they are found.
template <bool KS, bool TWO, bool SPLIT>
__device__ __forceinline__ void cta_giants(const Filter<3> &F, Match *list, uint32_t *keys, uint32_t *count, uint32_t cap,
                                           const uint32_t *ks, const uint16_t *rid, const uint32_t *__restrict__ row_k,
                                           uint32_t n, uint32_t warp, uint32_t warps, const GiantMul &G0,
                                           const GiantMul &G1, uint32_t s0) {
#pragma unroll 1
  for (uint32_t g = 4 * warp; g < n; g += 4 * warps) {
    uint32_t c[4];
    if (KS) {
      const uint4 v = *reinterpret_cast<const uint4 *>(ks + g);
      c[0] = v.x, c[1] = v.y, c[2] = v.z, c[3] = v.w;
    } else {
#pragma unroll
      for (uint32_t i = 0; i < 4; i++) c[i] = __ldg(row_k + rid[min(g + i, n - 1)]);
    }
    uint32_t hit = 0;
    auto rows = [&](auto count) {
#pragma unroll
      for (uint32_t i = 0; i < decltype(count)::value; i++) {
        if (F.test(giant_key<kRowsIntV>(c[i], G0, 0, 0, 0))) hit |= 1u << i;
        if (TWO && F.test(giant_key<kRowsIntV>(c[i], G1, 0, 0, 0))) hit |= 16u << i;
      }
    };
    if (SPLIT && n - g == 1) rows(std::integral_constant<uint32_t, 1>{});
    else if (SPLIT && n - g == 2) rows(std::integral_constant<uint32_t, 2>{});
    else rows(std::integral_constant<uint32_t, 4>{});
    if (hit) {  // rare
#pragma unroll 1
      for (uint32_t i = 0; i < 8; i++) {
        const uint32_t sl = g + (i & 3);
        if (!((hit >> i) & 1u) || sl >= n) continue;
        const GiantMul &G = i & 4 ? G1 : G0;
        const uint32_t k = KS ? ks[sl] : __ldg(row_k + rid[sl]);
        const uint64_t y = giant_exact<kRowsIntV>(k, G);
        uint32_t f;
        const bool edge = exact_key<kRowsIntV>(y, giant_key<kRowsIntV>(k, G, 0, 0, 0), G.p, 0, f);
        // (edge: a baby step may be stored under the next key)
        const uint32_t idx = atomicAdd(count, edge ? 2u : 1u);
        for (uint32_t e = 0; e <= (uint32_t)edge; e++)
          if (idx + e < cap) {
            list[idx + e] = Match{y, rid[sl], s0 + (i & 4 ? 32 : 0)};
            keys[idx + e] = f + e;
          }
      }
    }
  }
}

// The CTA-per-prime kernel, for jobs whose best baby-step count needs a filter
// larger than a warp's share of shared memory (many k, wide n ranges).  All
// kCtaWarps warps of a CTA work on one prime: thread t runs baby chains t and
// t + 32W into one filter that fills most of the SM's shared memory; the active
// rows are sorted by their residue r, and for each r the warps share the rows
// (32 lanes per row, T/32 steps per lane) with the lane's multiplier Z*b^r, so
// that every row is the integer k.  Shared memory:
//   [filter, fwords x 4 B][tags, 32W x chain_len x 4 B][k of the active rows,
//   row_slots x 4 B (when it fits: KS)][their row ids, row_slots x 2 B]
//   [match_cap suspects][their keys][rows per residue, Q x 4 B][count, redo flag, 16 B]
// What bounds it is the integer pipes, as the warp kernel, at four warps a
// scheduler.  On the wide job (1000 k, T = 64) it takes 103 ns per prime against 156
// with buckets of eight 16-bit tags, counts and signatures: giant steps 49 (one
// high product, one multiply-add and a 4-byte probe instead of a 32-bit Shoup
// product and a 16-byte probe), baby steps 19, suspects 18 (about 12 a prime),
// clearing and row lists 17 (25 before the next prime's loads were moved
// under the giant steps).  With shared memory for it two CTAs share an SM
// (CTAS, at 64 registers a thread): 467 k at m = 7168, T = 64 take 47 ns against 52.5.
// SPLIT: residues with rows for few of the 16 warps (JobDev::split) are gone through
// side by side, and a residue's steps by several warps in turn.  With all warps at one
// residue most have no row and form its multipliers only: two k over 2e8 exponents (Q =
// 48, T = 256, m = 16384) took 344 ns per prime, so split 92; twelve over 6e7 224, 92.
template <bool KS, int CTAS, bool SPLIT>
__global__ void __launch_bounds__(32 * kCtaWarps, CTAS) bsgs_cta_kernel(JobDev J, ChunkBufs cb, HitBufs hb) {
  extern __shared__ uint4 smem4[];
  constexpr uint32_t T = 32 * kCtaWarps;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t CL = J.chain_len, spl = J.steps_per_lane;
  uint32_t *fwords = reinterpret_cast<uint32_t *>(smem4);
  uint32_t *tags = fwords + J.fwords;
  uint32_t *ks = tags + T * CL;
  uint16_t *rid = reinterpret_cast<uint16_t *>(ks + (KS ? J.row_slots : 0));
  Match *list = reinterpret_cast<Match *>(rid + J.row_slots);
  uint32_t *keys = reinterpret_cast<uint32_t *>(list + J.match_cap);
  uint32_t *nrow = keys + J.match_cap;
  uint32_t *count = nrow + J.Q;
  Filter<3> F;
  F.w = fwords;
  F.sh1 = J.fshift;
  F.mul = J.fwords << J.fshift;
  const uint32_t total = *cb.count;
  const uint32_t n = total < cb.cap ? total : cb.cap;  // (the thread's chains begin at tid*CL and (tid + T)*CL; m == 2*T*CL)

  // What a prime needs first is loaded during the giant steps of the one before
  // it: its header and the thread's first two row ids with their k and slots.
  uint64_t np_ = 0, npinv = 0, nBl = 0;
  uint32_t nn = 0, nid[2] = {0, 0};
  uint2 nkr[2] = {};
  auto fetch = [&](uint32_t i) {
    const uint64_t *rec = cb.recs + (size_t)i * J.rec_elems;
    nn = (uint32_t)rec[kElNact];
    np_ = rec[kElP];
    npinv = rec[kElPinv];
    nBl = rec[J.el_tab + lane];
    const uint16_t *ids = reinterpret_cast<const uint16_t *>(rec + J.el_row);
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
      nid[h] = tid + h * T < nn ? ids[tid + h * T] : 0;
      nkr[h] = __ldg(J.row_kr + nid[h]);
    }
  };
  if (blockIdx.x < n) fetch(blockIdx.x);
#pragma unroll 1
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint64_t *rec = cb.recs + (size_t)i * J.rec_elems;
    const uint32_t nact = nn;
    if (nact == 0) {
      if (i + gridDim.x < n) fetch(i + gridDim.x);
      continue;
    }
    const uint64_t p = np_, pinv = npinv, np = 0 - p;
    uint64_t Bl = nBl;
    const uint64_t Stw = rec[kElStw], Stq = rec[kElStq];
    const uint64_t ofw = rec[kElOfw], ofq = rec[kElOfq];
    const uint64_t ww = rec[kElWoff + 2 * warp], wq = rec[kElWoff + 2 * warp + 1];
    if (i + gridDim.x < n && 16 * tid < J.rec_elems)  // the next prime's record into L2
      asm volatile("prefetch.global.L2 [%0];" ::"l"(rec + (size_t)gridDim.x * J.rec_elems + 16 * tid));
    __syncthreads();  // the previous prime is done with shared memory
    const uint4 z4 = make_uint4(0, 0, 0, 0);
#pragma unroll 4
    for (uint32_t q = tid; q < J.fwords / 4; q += T) smem4[q] = z4;
    for (uint32_t q = tid; q < J.Q + 2; q += T) nrow[q] = 0;  // and count and the redo flag
    __syncthreads();
    // the active rows into their residues' lists (in any order): x the k, y the residue's first slot and r
    auto place = [&](bool on, uint32_t id, uint2 kr) {
      const uint32_t r = on ? kr.y & 0xfffu : 0xffffffffu;
      const uint32_t same = __match_any_sync(0xffffffffu, r);
      const int lead = __ffs(same) - 1;
      uint32_t at = 0;
      if (on && (int)lane == lead) at = atomicAdd(&nrow[r], __popc(same));
      at = __shfl_sync(0xffffffffu, at, lead) + __popc(same & ((1u << lane) - 1u)) + (kr.y >> 12);
      if (!on) return;
      rid[at] = (uint16_t)id;
      if (KS) ks[at] = kr.x;
    };
    if (32 * warp < nact) place(tid < nact, nid[0], nkr[0]);
    if (32 * warp + T < nact) place(tid + T < nact, nid[1], nkr[1]);
#pragma unroll 1
    for (uint32_t a = tid + 2 * T; a < ((nact + 31) & ~31u); a += T) {
      const uint32_t id = a < nact ? reinterpret_cast<const uint16_t *>(rec + J.el_row)[a] : 0;
      place(a < nact, id, __ldg(J.row_kr + id));
    }

    // Baby steps: chain starts B^(lane*c) times the warp's offset B^(32w*c)
    if (warp) Bl = shoup_mul(Bl, ww, wq, p);
    const uint64_t Blb = shoup_mul(Bl, ofw, ofq, p);
    if (cb.small_step == kStepShoup)
      baby_filter<true, true, 4>(F, tags + tid, T, J.edge_lim, Bl, Blb, CL, CL, CL, pinv, LazyShoup{Stw, Stq, np});
    else
      baby_filter<true, true, 4>(F, tags + tid, T, J.edge_lim, Bl, Blb, CL, CL, CL, pinv,
                                 LazyShort{J.bq_small, (uint32_t)(Stq >> (32 - cb.step_shift)), cb.step_shift, np});
    __syncthreads();

    // Giant steps, residue by residue: the multiplier's stored form E = Z*b^r
    {
      const uint64_t bw = rec[kElWoff + 2 * kCtaWarps], bq = rec[kElWoff + 2 * kCtaWarps + 1];
      const uint64_t Gw = rec[kElGw], Gq = rec[kElGq];
      uint64_t Er = rec[J.el_tab + 32 + lane];
      if (i + gridDim.x < n) fetch(i + gridDim.x);
      if constexpr (SPLIT) {
        // The warp's place (slot) goes through residues slots apart, one of the pair r0,
        // r0 + 1 and the other by turns: for even Q the active rows of few k are of one parity.
        const uint32_t ws = J.split & 255, slots = J.split >> 8 & 255, wsteps = J.split >> 16;
        const uint32_t slot = warp / (ws * wsteps), wr = warp % ws, wu = warp / ws % wsteps;
        const uint32_t r0 = slots > 1 ? slot & ~1u : slot;
        uint64_t pw = bw, pq = bq;  // b^slots and its Shoup constant, by squarings; b^r0 into Er
#pragma unroll 1
        for (uint32_t x = r0, y = slots; y > 1; x >>= 1, y >>= 1) {
          if (x & 1) Er = shoup_mul(Er, pw, pq, p);
          const uint64_t sq = shoup_mul(pq * np, pw, pq, p);  // (pq * np is pw in Montgomery form)
          pw = shoup_mul(pw, pw, pq, p);
          pq = shoup_const(sq, pinv);
        }
#pragma unroll 1
        for (uint32_t rb = r0, turn = slot; slot < slots && rb < J.Q; rb += slots, turn++) {
          const uint32_t r = slots > 1 ? rb + (turn & 1) : rb;
          const uint32_t nr = r < J.Q ? nrow[r] : 0;
          if (nr) {
            const uint32_t at = __ldg(J.row_base + r);
            uint64_t E = r != rb ? shoup_mul(Er, bw, bq, p) : Er;
#pragma unroll 1
            for (uint32_t u = 0; u < spl; u += 2) {
              const bool mine = (u >> 1) % wsteps == wu;
              GiantMul G0, G1;
              if (mine) G0.set(E, p, pinv);
              G1 = G0;
              if (u + 1 < spl) {
                E = shoup_mul(E, Gw, Gq, p);
                if (mine) {
                  G1.set(E, p, pinv);
                  cta_giants<KS, true, SPLIT>(F, list, keys, count, J.match_cap, ks + at, rid + at, J.row_k, nr, wr, ws, G0, G1, lane + 1 + 32 * u);
                }
                if (u + 2 < spl) E = shoup_mul(E, Gw, Gq, p);
              } else if (mine) {
                cta_giants<KS, false, SPLIT>(F, list, keys, count, J.match_cap, ks + at, rid + at, J.row_k, nr, wr, ws, G0, G1, lane + 1 + 32 * u);
              }
            }
          }
          Er = shoup_mul(Er, pw, pq, p);
        }
      } else {
#pragma unroll 1
        for (uint32_t r = 0; r < J.Q; r++) {
          const uint32_t nr = nrow[r];
          if (nr) {
            const uint32_t at = __ldg(J.row_base + r);
            const uint32_t w = (warp + 5 * r) % kCtaWarps;  // uneven shares of several residues fall on different warps
            uint64_t E = Er;
#pragma unroll 1
            for (uint32_t u = 0; u < spl; u += 2) {
              GiantMul G0, G1;
              G0.set(E, p, pinv);
              G1 = G0;
              if (u + 1 < spl) {
                E = shoup_mul(E, Gw, Gq, p);
                G1.set(E, p, pinv);
                cta_giants<KS, true, SPLIT>(F, list, keys, count, J.match_cap, ks + at, rid + at, J.row_k, nr, w, kCtaWarps, G0, G1, lane + 1 + 32 * u);
                if (u + 2 < spl) E = shoup_mul(E, Gw, Gq, p);
              } else {
                cta_giants<KS, false, SPLIT>(F, list, keys, count, J.match_cap, ks + at, rid + at, J.row_k, nr, w, kCtaWarps, G0, G1, lane + 1 + 32 * u);
              }
            }
          }
          if (r + 1 < J.Q) Er = shoup_mul(Er, bw, bq, p);
        }
      }
    }
    __syncthreads();

    // Suspects, eight at a time: each thread scans its own tags (its two chains,
    // 16 bits of each value's key) for their exact keys.  Tag matches (about three
    // a prime on the wide job, nearly all false) go to settle_kernel: a thread that
    // walked its chains here kept the whole CTA waiting, 17 of 117 ns per prime.
    const uint32_t mc = *count;
    if (mc > J.match_cap) {
      if (tid == 0) {
        const uint32_t r = atomicAdd(cb.redo_count, 1u);
        if (r < cb.cap) cb.redo[r] = i;
      }
      continue;
    }
#pragma unroll 1
    for (uint32_t q0 = 0; q0 < mc; q0 += 8) {
      uint32_t tag[8], z[8];
#pragma unroll
      for (uint32_t q = 0; q < 8; q++) {
        tag[q] = __byte_perm(keys[min(q0 + q, mc - 1)], 0, 0x1010);
        z[q] = 0xffffffffu;
      }
#pragma unroll 4
      for (uint32_t t = 0; t < CL; t++) {
        const uint32_t tp = tags[t * T + tid];
#pragma unroll
        for (uint32_t q = 0; q < 8; q++) z[q] = __vminu2(z[q], tp ^ tag[q]);
      }
      uint32_t hit = 0;
#pragma unroll
      for (uint32_t q = 0; q < 8; q++) hit |= zero_half(z[q]) && q0 + q < mc ? 1u << q : 0u;
#pragma unroll 1
      for (; hit; hit &= hit - 1) {
        const Match mt = list[q0 + __ffs(hit) - 1];
        const uint32_t idx = atomicAdd(cb.redo_count + 1, 1u);
        if (idx < cb.cand_cap) {
          cb.cand[idx] = Candidate{mt.y, i, mt.row, mt.s, tid};
        } else if (atomicExch(count + 1, 1u) == 0) {  // no room: the exact path takes the prime, once
          const uint32_t r = atomicAdd(cb.redo_count, 1u);
          if (r < cb.cap) cb.redo[r] = i;
        }
      }
    }
  }
}

// The tag matches of a CTA launch: one thread per candidate walks the two baby
// chains of the thread that found it and compares the values themselves.
__global__ void __launch_bounds__(128) settle_kernel(JobDev J, ChunkBufs cb, HitBufs hb) {
  const uint32_t cnt = cb.redo_count[1], n = cnt < cb.cand_cap ? cnt : cb.cand_cap;
  const uint32_t T = 32 * J.cta_warps, CL = J.chain_len;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    const Candidate x = cb.cand[c];
    const uint64_t *rec = cb.recs + (size_t)x.i * J.rec_elems;
    const uint64_t p = rec[kElP], pinv = rec[kElPinv], Stw = rec[kElStw], Stq = rec[kElStq];
    const uint32_t w = x.thread >> 5;
    uint64_t va = rec[J.el_tab + (x.thread & 31)];
    if (w) va = shoup_mul(va, rec[kElWoff + 2 * w], rec[kElWoff + 2 * w + 1], p);
    uint64_t vb = shoup_mul(va, rec[kElOfw], rec[kElOfq], p);
    va = from_mont(va, p, pinv);
    vb = from_mont(vb, p, pinv);
#pragma unroll 1
    for (uint32_t t = 0; t < CL; t++) {
      if (va == x.y) record_hit(J, hb, p, x.row, x.s, x.thread * CL + t);
      if (vb == x.y) record_hit(J, hb, p, x.row, x.s, (x.thread + T) * CL + t);
      va = shoup_mul(va, Stw, Stq, p);
      vb = shoup_mul(vb, Stw, Stq, p);
    }
  }
}

// The exact path: a table of (tag << jbits) | j entries with linear probing per
// prime, for the primes with too many suspects for the fast path.  WG
// warps share a prime (1 for warp-per-prime jobs, kCtaWarps for CTA jobs) with
// the same chain layout as the fast kernels.
// The smallest primes come here, and among them those modulo which B has a small
// order d: their baby steps are d values over and over.  The table holds the first
// d, and a match stands for j, j + d, ...; all m of them made runs of m/d
// entries in one place of the table, which each insert and probe walked.
template <int WG>
__global__ void __launch_bounds__(WG == 1 ? 32 * kWarpsPerBlock : 32 * WG, 1)
bsgs_exact_kernel(JobDev J, ChunkBufs cb, HitBufs hb) {
  extern __shared__ uint4 smem4[];
  constexpr uint32_t G = 32 * WG;                           // threads per prime
  constexpr uint32_t NG = WG == 1 ? kWarpsPerBlock : 1;     // primes per block
  __shared__ uint32_t order;  // WG > 1
  const uint32_t grp = threadIdx.x / G, gt = threadIdx.x % G, wig = gt >> 5, lane = threadIdx.x & 31;
  const uint32_t S = 1u << J.exact_log2;
  const uint32_t tmask = S - 1;
  // the table in shared memory, or (tables larger than shared memory) in this
  // CTA's slice of the chunk's global scratch
  uint32_t *tab = (J.exact_global ? cb.exact_tab + (size_t)blockIdx.x * NG * S : reinterpret_cast<uint32_t *>(smem4)) +
                  (size_t)grp * S;
  const uint32_t jbits = J.jbits;
  const uint32_t jmask = (1u << jbits) - 1u;
  const uint32_t tagmask = (1u << (32 - jbits)) - 1u;
  const uint32_t tl = J.exact_log2;
  const uint32_t lane_t = lane & (J.tlanes - 1);
  const uint32_t lane_row = lane / J.tlanes;
  const uint32_t rows_pass = J.rows_per_it * WG;  // row slots per pass of the group
  const uint32_t rc = *cb.redo_count;
  const bool all = rc > cb.cap;  // more entries than the list holds: every prime of the chunk
  const uint32_t nr = !all ? rc : *cb.count < cb.cap ? *cb.count : cb.cap;
  const uint32_t ngroups = gridDim.x * NG;
  if (blockIdx.x == 0 && threadIdx.x == 0 && nr) atomicAdd(&hb.stat[kStatExact], (unsigned long long)nr);
#pragma unroll 1
  for (uint32_t r = blockIdx.x * NG + grp; r < nr; r += ngroups) {
    const uint32_t i = all ? r : cb.redo[r];
    const uint64_t p = rec_el(J, cb, kElP, i), pinv = rec_el(J, cb, kElPinv, i);
    const uint32_t nact = (uint32_t)rec_el(J, cb, kElNact, i);
    const uint64_t Gs = rec_el(J, cb, kElGs, i);
    const uint64_t Stw = rec_el(J, cb, kElStw, i), Stq = rec_el(J, cb, kElStq, i);
    if (WG == 1) __syncwarp();
    else __syncthreads();
    for (uint32_t q = gt; q < S; q += G) tab[q] = kEmpty;
    if (WG > 1 && gt == 0) order = J.m;
    if (WG == 1) __syncwarp();
    else __syncthreads();
    // the thread's two baby chains, j = (gt + G*c)*chain_len + t
    uint64_t Bl = rec_el(J, cb, J.el_tab + lane, i);
    if (WG > 1 && wig) Bl = shoup_mul(Bl, rec_el(J, cb, kElWoff + 2 * wig, i), rec_el(J, cb, kElWoff + 2 * wig + 1, i), p);
    const uint64_t Blb = shoup_mul(Bl, rec_el(J, cb, kElOfw, i), rec_el(J, cb, kElOfq, i), p);
    // the first j at which the values repeat the one of j = 0, or m
    uint32_t d = J.m;
    {
      const uint64_t v0 = rec_el(J, cb, J.el_tab, i);
#pragma unroll 1
      for (uint32_t c = 0; c < 2; c++) {
        const uint32_t j0 = (gt + G * c) * J.chain_len;
        uint64_t v = c ? Blb : Bl;
#pragma unroll 1
        for (uint32_t j = j0; j < d && j < j0 + J.chain_len; j++) {
          if (v == v0 && j) d = j;
          v = shoup_mul(v, Stw, Stq, p);
        }
      }
      if (WG == 1) {
        d = __reduce_min_sync(0xffffffffu, d);
      } else {
        if (d < J.m) atomicMin(&order, d);
        __syncthreads();
        d = order;
      }
    }
#pragma unroll 1
    for (uint32_t c = 0; c < 2; c++) {
      const uint32_t j0 = (gt + G * c) * J.chain_len;
      uint64_t v = c ? Blb : Bl;
      if (J.int_rows) v = from_mont(v, p, pinv);  // giant values (below) come in normal form
#pragma unroll 1
      for (uint32_t j = j0; j < d && j < j0 + J.chain_len; j++) {
        uint32_t h = (uint32_t)v & tmask;
        const uint32_t e = ((((uint32_t)(v >> tl)) & tagmask) << jbits) | j;
#pragma unroll 1
        for (uint32_t t = 0; t < S; t++) {
          if (atomicCAS(&tab[h], kEmpty, e) == kEmpty) break;
          h = (h + 1) & tmask;
        }
        v = shoup_mul(v, Stw, Stq, p);
      }
    }
    if (WG == 1) __syncwarp();
    else __syncthreads();
    const uint64_t Gl = rec_el(J, cb, J.el_tab + 32 + lane, i);
    const uint32_t ngi = (nact + rows_pass - 1) / rows_pass;
#pragma unroll 1
    for (uint32_t gi = 0; gi < ngi; gi++) {
      const uint32_t slot = gi * rows_pass + wig * J.rows_per_it + lane_row;
      if (slot < nact) {
        const uint32_t row = J.row_mask ? nth_row(rec_el(J, cb, J.el_v, i), slot)
                                        : (uint32_t)(rec_el(J, cb, J.el_row + (slot >> 2), i) >> (16 * (slot & 3))) &
                                              0xffffu;
        // integer rows: the normal form of k*b^r*Z from Z's Montgomery form (CTA layout
        // and by_res, whose k*b^r may exceed 32 bits: k*Z, times b per residue step)
        uint64_t y;
        if (WG > 1 || J.by_res) {
          y = montmul((uint64_t)__ldg(J.row_k + row), Gl, p, pinv);
          constexpr uint32_t eb = WG > 1 ? kElWoff + 2 * WG : kElV;
          const uint64_t bw = rec_el(J, cb, eb, i), bq = rec_el(J, cb, eb + 1, i);
#pragma unroll 1
          for (uint32_t q = __ldg(J.row_r + row); q; q--) y = shoup_mul(y, bw, bq, p);
        } else {
          y = montmul(J.row_ids_only || J.row_mask ? (uint64_t)__ldg(J.row_c + row) : rec_el(J, cb, J.el_v + slot, i), Gl,
                      p, pinv);
        }
        uint32_t s = lane_t + 1;
#pragma unroll 1
        for (uint32_t u = 0; u < J.steps_per_lane; u++) {
          uint32_t h = (uint32_t)y & tmask;
          const uint32_t tag = ((uint32_t)(y >> tl)) & tagmask;
#pragma unroll 1
          for (uint32_t q = 0; q < S; q++) {
            const uint32_t e = tab[h];
            if (e == kEmpty) break;
            if ((e >> jbits) == tag)
              for (uint32_t j = e & jmask; j < J.m; j += d) record_hit(J, hb, p, row, s, j);
            h = (h + 1) & tmask;
          }
          if (u + 1 < J.steps_per_lane) {
            y = montmul(y, Gs, p, pinv);
            s += 32;
          }
        }
      }
    }
  }
}

int bsgs_exact_smem_bytes(const JobDev &job) {
  return job.exact_global ? 0 : (job.cta_warps > 1 ? 1 : kWarpsPerBlock) * (4 << job.exact_log2);
}

uint64_t bsgs_exact_scratch_bytes(const JobDev &job, int exact_grid) {
  if (!job.exact_global) return 0;
  return (uint64_t)exact_grid * (job.cta_warps > 1 ? 1 : kWarpsPerBlock) * (4ull << job.exact_log2);
}

static cudaError_t configure_one(const void *fn, int smem, int threads, int device, int *grid_out) {
  // The limit is a property of the kernel shared by every job in the process,
  // so it is set to the device maximum (the same value from every thread)
  // rather than to this job's size, which a concurrent job could lower.
  int max_smem = 0;
  cudaError_t e = cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (e != cudaSuccess) return e;
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, fn);
  if (e != cudaSuccess) return e;
  max_smem -= (int)fa.sharedSizeBytes;  // the kernel's static shared memory counts against the same limit
  if (smem > max_smem) return cudaErrorInvalidValue;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
  if (e != cudaSuccess) return e;
  int sms = 0;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  *grid_out = per_sm * sms;
  return cudaSuccess;
}

static int bsgs_threads(const JobDev &job) { return job.cta_warps > 1 ? 32 * kCtaWarps : 32 * kWarpsPerBlock; }

static BsgsFn bsgs_cta_fn(const JobDev &job) {
  // (cta_pair leaves room for the rows' k)
  if (job.split) {
    if (job.cta_pair) return bsgs_cta_kernel<true, 2, true>;
    return job.ctab_smem ? bsgs_cta_kernel<true, 1, true> : bsgs_cta_kernel<false, 1, true>;
  }
  if (job.cta_pair) return bsgs_cta_kernel<true, 2, false>;
  return job.ctab_smem ? bsgs_cta_kernel<true, 1, false> : bsgs_cta_kernel<false, 1, false>;
}

static const void *bsgs_fast_fn(const JobDev &job) {
  if (job.cta_warps > 1) return (const void *)bsgs_cta_fn(job);
  return (const void *)bsgs_fn(job);
}

static const void *bsgs_exact_fn(const JobDev &job) {
  return job.cta_warps > 1 ? (const void *)bsgs_exact_kernel<kCtaWarps> : (const void *)bsgs_exact_kernel<1>;
}

cudaError_t bsgs_configure(const JobDev &job, int device, int *grid_out, int *exact_grid_out) {
  cudaError_t e = configure_one(bsgs_fast_fn(job), bsgs_smem_bytes(job), bsgs_threads(job), device, grid_out);
  if (e != cudaSuccess) return e;
  e = configure_one(bsgs_exact_fn(job), bsgs_exact_smem_bytes(job), bsgs_threads(job), device, exact_grid_out);
  if (e != cudaSuccess) return e;
  if (job.exact_global) {  // one CTA per SM keeps the global scratch small (the exact path is rare)
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess && sms > 0 && *exact_grid_out > sms) *exact_grid_out = sms;
  }
  return e;
}

cudaError_t launch_bsgs(const JobDev &job, const ChunkBufs &cb, const HitBufs &hb, int grid,
                        cudaStream_t st) {
  if (job.cta_warps > 1)
  {
    bsgs_cta_fn(job)<<<grid, 32 * kCtaWarps, bsgs_smem_bytes(job), st>>>(job, cb, hb);
    settle_kernel<<<grid, 128, 0, st>>>(job, cb, hb);
  } else
    bsgs_fn(job)<<<grid, 32 * kWarpsPerBlock, bsgs_smem_bytes(job), st>>>(job, cb, hb);
  return cudaGetLastError();
}

static BatchFn batch_fn(const JobDev &rep) {
  switch (row_mode(rep)) {
    case kRowsFew: return bsgs_batch_kernel<32, kRowsFew>;
    case kRowsRes: return batch_fn_t<kRowsRes>(rep.tlanes);
    case kRowsMask: return batch_fn_t<kRowsMask>(rep.tlanes);
    case kRowsIntId: return batch_fn_t<kRowsIntId>(rep.tlanes);
    case kRowsIntV: return batch_fn_t<kRowsIntV>(rep.tlanes);
    default: return batch_fn_t<kRowsV>(rep.tlanes);
  }
}


cudaError_t batch_configure(const JobDev &rep, uint32_t warp_bytes, int device, int *grid_out) {
  return configure_one((const void *)batch_fn(rep), kWarpsPerBlock * (int)warp_bytes, 32 * kWarpsPerBlock, device,
                       grid_out);
}

cudaError_t launch_bsgs_batch(const JobDev &rep, const BatchItem *items, uint32_t nitems, uint32_t stage_max,
                              uint32_t row_slots_max, uint32_t warp_bytes, int grid, cudaStream_t st) {
  if (nitems == 0) return cudaSuccess;
  if (nitems > kBatchMaxItems) return cudaErrorInvalidValue;
  batch_fn(rep)<<<grid, 32 * kWarpsPerBlock, kWarpsPerBlock * warp_bytes, st>>>(items, nitems, warp_bytes, stage_max,
                                                                                       row_slots_max);
  return cudaGetLastError();
}

cudaError_t launch_bsgs_exact(const JobDev &job, const ChunkBufs &cb, const HitBufs &hb, int grid,
                              cudaStream_t st) {
  if (job.cta_warps > 1)
    bsgs_exact_kernel<kCtaWarps><<<grid, 32 * kCtaWarps, bsgs_exact_smem_bytes(job), st>>>(job, cb, hb);
  else
    bsgs_exact_kernel<1><<<grid, 32 * kWarpsPerBlock, bsgs_exact_smem_bytes(job), st>>>(job, cb, hb);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Direct verification of every candidate hit.

__global__ void verify_kernel(JobDev J, HitBufs hb) {
  const uint32_t cnt = *hb.raw_count;
  const uint32_t n = cnt < hb.cap ? cnt : hb.cap;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const Hit h = hb.raw[i];
    const uint64_t p = h.p;
    Mont M;
    M.p = p;
    M.pinv = mont_pinv(p);
    uint64_t one, r2;
    mont_consts(p, M.pinv, one, r2);
    const uint64_t bmod = p > J.base ? (uint64_t)J.base : (uint64_t)J.base % p;
    const uint64_t bm = montmul(bmod, r2, M);
    const uint64_t x = mont_pow(bm, h.n, one, M);
    const uint64_t km = montmul((uint64_t)h.k, r2, M);
    const uint64_t y = montmul(montmul(x, km, M), 1, M);  // k*b^n mod p, normal form
    const uint64_t want = J.sign < 0 ? 1 : p - 1;
    if (y == want) {
      const uint32_t idx = atomicAdd(hb.fac_count, 1u);
      if (idx < hb.cap) hb.fac[idx] = h;
    }
  }
}

cudaError_t launch_verify(const JobDev &job, const HitBufs &hb, cudaStream_t st) {
  const unsigned blocks = std::min(4 * kSms, (hb.cap + 255) / 256);  // (grid-stride)
  verify_kernel<<<blocks, 256, 0, st>>>(job, hb);
  return cudaGetLastError();
}

}  // namespace rs
