// Rice (format 2) encoder on the GPU: BF16 words already on the device -> the file arrays
// (raw, meta, bits, roff), bit for bit what the host encoder and the reference's
// binade/rice.py:57-125 write. The reference encodes on the CPU with numpy (about a million
// weights a second); this is three passes over the tensor at memory speed.
//
//   bn_bf16_split_hist   raw byte (sign << 7 | mantissa) of every word and the histogram of the
//                        exponent bytes
//   bn_rank_table        the rank table of a histogram (binade/format.py:34-42)
//   bn_rice_encode_plan  per tile the Rice parameter k (0..3) with the smallest cost
//                        k n + sum min(q + 1, qmax), q = rank >> k, qmax = max q <= 63, ties to the
//                        smaller k (binade/rice.py:57-73) -> meta = k | qmax << 2; per row the
//                        stream's length in 32-bit words; then the rows' first words (exclusive
//                        prefix sum) and the total
//   bn_rice_encode_write the streams
//
// Plan and write take a tile per thread: a warp looks the ranks of 32 tiles up with eight lanes per
// tile (16 weights a lane), leaves them in shared memory as bytes, and every thread transposes
// its tile's 128 bytes to eight bit planes in registers. From there a cost is a few population
// counts, the plane of the weights with q > j a logical operation, and a unary plane the bits of
// one mask at the set positions of another, packed eight weights at a time through a table.
// With a warp per tile (a lane holding four weights, one prefix sum over the lanes per plane)
// plan and write took 115 and 384 us on 15360 x 3840; now 43 and 112. Bound: instruction issue (1570
// and 3860 warp instructions for the 30 tiles of a row, of which looking the ranks up and turning
// them into bit planes about 1200).
#include "rice.cuh"

namespace bn {
namespace {

constexpr int HIST_THREADS = 512;

// Eight words a thread and step; the histogram has a copy per lane (a lane's copies never share a
// bank, and nearly all weights fall into a handful of bins, where one copy per block made the
// lanes of a warp wait for each other). Bound: the shared atomics; 15360 x 3840: 48.6 us with one
// word a step and one copy, now 40 (HBM would take 27).
__global__ void __launch_bounds__(HIST_THREADS) split_hist_kernel(const uint16_t *__restrict__ w, int64_t n, uint8_t *__restrict__ raw, uint32_t *__restrict__ hist, bool aligned) {
  __shared__ uint32_t h[256 * 32];
  for (int i = threadIdx.x; i < 256 * 32; i += HIST_THREADS) h[i] = 0;
  __syncthreads();
  uint32_t *const mine = h + lane_id();
  auto count = [&](uint32_t v) { atomicAdd(mine + ((v >> 7) & 0xFFu) * 32u, 1u); };
  const int64_t step = (int64_t)gridDim.x * HIST_THREADS, first = (int64_t)blockIdx.x * HIST_THREADS + threadIdx.x;
  const int64_t eights = aligned ? n / 8 : 0;
  auto take = [&](uint4 v, int64_t i) {
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
    uint32_t r[2];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      count(x[j] & 0xFFFFu), count(x[j] >> 16);
      const uint32_t b = ((x[j] >> 8) & 0x00800080u) | (x[j] & 0x007F007Fu);  // two raw bytes, in bytes 0 and 2
      if (j & 1) r[j >> 1] |= __byte_perm(b, 0u, 0x2044);
      else r[j >> 1] = __byte_perm(b, 0u, 0x4420);
    }
    *reinterpret_cast<uint2 *>(raw + i * 8) = make_uint2(r[0], r[1]);
  };
  int64_t i = first;
  for (; i + step < eights; i += 2 * step) {  // two loads in flight
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(w) + i), u = __ldg(reinterpret_cast<const uint4 *>(w) + i + step);
    take(v, i), take(u, i + step);
  }
  if (i < eights) take(__ldg(reinterpret_cast<const uint4 *>(w) + i), i);
  for (int64_t j = eights * 8 + first; j < n; j += step) {
    const uint32_t v = w[j];
    raw[j] = (uint8_t)(((v >> 8) & 0x80u) | (v & 0x7Fu));
    count(v);
  }
  __syncthreads();
  for (int bin = threadIdx.x >> 5; bin < 256; bin += HIST_THREADS / 32) {
    const uint32_t sum = __reduce_add_sync(BN_FULL, h[bin * 32 + lane_id()]);
    if (lane_id() == 0 && sum) atomicAdd(hist + bin, sum);
  }
}

// Exponents by descending count, equal counts by ascending exponent; those that never occur are
// listed as 0 (binade/format.py:34-42). One thread per exponent. On the host the table cost a
// read of the histogram and two copies back, each with a synchronisation.
__global__ void __launch_bounds__(256) rank_table_kernel(const uint32_t *__restrict__ hist, uint8_t *__restrict__ table, uint8_t *__restrict__ rank) {
  __shared__ uint32_t h[256];
  const uint32_t e = threadIdx.x, own = hist[e];
  h[e] = own;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t i = 0; i < 256; i++) before += h[i] > own || (h[i] == own && i < e);
  rank[e] = (uint8_t)before, table[before] = own ? (uint8_t)e : 0u;
}

// ---------------------------------------------------------------------------------------------
// A warp's 32 tiles as bit planes
// ---------------------------------------------------------------------------------------------
constexpr int EN_WARPS = 28;                  // of the plan
constexpr int EN_WRITE_WARPS = 20;            // of the write: its planes, low planes and masks take 90 registers
constexpr uint32_t EN_TILE = 36;              // words between two tiles' ranks in shared memory: 32, and no bank conflicts for 16-byte accesses
constexpr uint32_t EN_WORDS = 32 * EN_TILE;   // words of a warp's ranks
constexpr uint32_t EN_WINDOW = 512;           // words of the stream a warp puts together at a time (a tile touches at most 266)
constexpr uint32_t EN_PACK = 65536;           // byte [value | alive << 8]: the bits of `value` at the set positions of `alive`, packed
constexpr uint32_t EN_SMEM = EN_PACK + 512 + EN_WRITE_WARPS * (EN_WORDS + EN_WINDOW) * 4;
constexpr uint32_t EN_FEW = 8;                // alive weights up to which a plane is one lookup

// The tiles of a task of whole rows (several when 32 tiles hold them): lane -> (row, tile).
struct EncTask {
  int64_t row0;
  int rows, rows_per_task, t0, count;  // rows of the task, first tile of the chunk, its tiles
};
struct EncSource {
  const uint16_t *w;
  int64_t K;
  int T;
  bool wide;  // rows of whole 16-byte pieces, aligned
};

// Ranks of the chunk's tiles into sh (128 bytes a tile; weights past a row's end: rank 0), then bit
// plane b of this lane's tile in r[b]. Whole warp calls it.
__device__ __forceinline__ void tile_planes(const EncSource &src, const EncTask &task, const uint8_t *rank, uint32_t *sh, uint32_t lane, int sub, int t, uint32_t (&r)[8][4]) {
  for (int u0 = 0; u0 < task.count; u0 += 4) {
    const int u = u0 + (int)(lane >> 3);
    const int us = __shfl_sync(BN_FULL, sub, u & 31), ut = __shfl_sync(BN_FULL, t, u & 31);
    if (u >= task.count) continue;
    const int64_t col = (int64_t)ut * BN_TILE + (lane & 7u) * 16;
    const int left = (int)min((int64_t)16, src.K - col);  // weights of this lane inside the row
    const uint16_t *const p = src.w + (task.row0 + us) * src.K + col;
    uint32_t x[8];
    if (src.wide && left == 16) {
      const uint4 a = __ldg(reinterpret_cast<const uint4 *>(p)), b = __ldg(reinterpret_cast<const uint4 *>(p) + 1);
      x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w, x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t lo = 2 * i < left ? p[2 * i] : 0u, hi = 2 * i + 1 < left ? p[2 * i + 1] : 0u;
        x[i] = lo | (hi << 16);
      }
    }
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t r0 = rank[(x[2 * i] >> 7) & 0xFFu], r1 = rank[(x[2 * i] >> 23) & 0xFFu], r2 = rank[(x[2 * i + 1] >> 7) & 0xFFu], r3 = rank[(x[2 * i + 1] >> 23) & 0xFFu];
      o[i] = r0 | (r1 << 8) | (r2 << 16) | (r3 << 24);
    }
    if (left < 16) {
#pragma unroll
      for (int i = 0; i < 4; i++) o[i] &= low_mask(8 * (left - 4 * i));
    }
    *reinterpret_cast<uint4 *>(sh + u * EN_TILE + (lane & 7u) * 4) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; i++) {
    uint32_t v[8];  // 32 ranks: word g holds weights 4g .. 4g + 3
    const uint4 a = *reinterpret_cast<const uint4 *>(sh + lane * EN_TILE + i * 8), b = *reinterpret_cast<const uint4 *>(sh + lane * EN_TILE + i * 8 + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    uint32_t even[4], odd[4];  // byte j of the words with even and with odd g
    auto bytes = [](uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&x)[4]) {
      const uint32_t l0 = __byte_perm(a, b, 0x5140), h0 = __byte_perm(a, b, 0x7362), l1 = __byte_perm(c, d, 0x5140), h1 = __byte_perm(c, d, 0x7362);
      x[0] = __byte_perm(l0, l1, 0x5410), x[1] = __byte_perm(l0, l1, 0x7632), x[2] = __byte_perm(h0, h1, 0x5410), x[3] = __byte_perm(h0, h1, 0x7632);
    };
    bytes(v[0], v[2], v[4], v[6], even), bytes(v[1], v[3], v[5], v[7], odd);
    auto swap = [](uint32_t &x, uint32_t &y, int sh, uint32_t mask) {
      const uint32_t t = ((x >> sh) ^ y) & mask;
      y ^= t, x ^= t << sh;
    };
#pragma unroll
    for (int half = 0; half < 2; half++) {  // the ranks' lower and upper four bits
      uint32_t n[4];                        // nibble g of n[j]: that half of weight 4g + j
#pragma unroll
      for (int j = 0; j < 4; j++) n[j] = half ? ((even[j] >> 4) & 0x0F0F0F0Fu) | (odd[j] & 0xF0F0F0F0u) : (even[j] & 0x0F0F0F0Fu) | ((odd[j] << 4) & 0xF0F0F0F0u);
      swap(n[0], n[2], 2, 0x33333333u), swap(n[1], n[3], 2, 0x33333333u);
      swap(n[0], n[1], 1, 0x55555555u), swap(n[2], n[3], 1, 0x55555555u);
#pragma unroll
      for (int j = 0; j < 4; j++) r[4 * half + j][i] = n[j];
    }
  }
  __syncwarp();
}

// What a warp's lanes work on, chunk by chunk of at most 32 tiles.
template <class Body>
__device__ __forceinline__ void each_task(int64_t R, int T, int rows_per_task, uint32_t warp, uint32_t lane, Body &&body) {
  const int64_t tasks = (R + rows_per_task - 1) / rows_per_task;
  for (int64_t i = (int64_t)warp * gridDim.x + blockIdx.x; i < tasks; i += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    EncTask task{i * rows_per_task, (int)min((int64_t)rows_per_task, R - i * rows_per_task), rows_per_task, 0, 0};
    for (; task.t0 < T; task.t0 += 32) {
      task.count = rows_per_task > 1 ? task.rows * T : min(32, T - task.t0);
      const bool mine = (int)lane < task.count;
      const int sub = mine && rows_per_task > 1 ? (int)lane / T : 0;
      body(task, mine, sub, mine ? (rows_per_task > 1 ? (int)lane - sub * T : task.t0 + (int)lane) : 0);
      if (rows_per_task > 1) break;
    }
  }
}

// Inclusive sum over the lanes of this lane's row (several rows a warp: T tiles each, else all lanes).
__device__ __forceinline__ uint32_t row_scan(uint32_t v, uint32_t lane, int t, int rows_per_task) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t n = __shfl_up_sync(BN_FULL, v, d);
    if (lane >= (uint32_t)d && (rows_per_task == 1 || t >= d)) v += n;
  }
  return v;
}

__global__ void __launch_bounds__(EN_WARPS * 32, 1) plan_kernel(EncSource src, const uint8_t *__restrict__ rank_table, int64_t R, int rows_per_task, uint8_t *__restrict__ meta, uint32_t *__restrict__ row_words) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t *const rank = smem;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t *const sh = reinterpret_cast<uint32_t *>(smem + 256) + warp * EN_WORDS;
  if (threadIdx.x < 256) rank[threadIdx.x] = rank_table[threadIdx.x];
  __syncthreads();
  uint64_t row_bits = 0;  // of the tiles before this chunk (one row a task)
  each_task(R, src.T, rows_per_task, warp, lane, [&](const EncTask &task, bool mine, int sub, int t) {
    uint32_t r[8][4];
    tile_planes(src, task, rank, sh, lane, sub, t, r);
    const int64_t n64 = src.K - (int64_t)t * BN_TILE;
    const uint32_t n = (uint32_t)min((int64_t)BN_TILE, n64);
    // the largest rank, and the weights whose rank equals it in the bits seen so far: after bit k
    // those with q == qmax
    uint32_t top[4], rmax = 0, at_top[4], sum[8];
#pragma unroll
    for (int i = 0; i < 4; i++) top[i] = low_mask((int)n - 32 * i);
#pragma unroll
    for (int b = 7; b >= 0; b--) {
      const uint32_t any = (top[0] & r[b][0]) | (top[1] & r[b][1]) | (top[2] & r[b][2]) | (top[3] & r[b][3]);
      if (any) {
        rmax |= 1u << b;
#pragma unroll
        for (int i = 0; i < 4; i++) top[i] &= r[b][i];
      }
      sum[b] = __popc(r[b][0]) + __popc(r[b][1]) + __popc(r[b][2]) + __popc(r[b][3]);
      if (b < 4) at_top[b] = __popc(top[0]) + __popc(top[1]) + __popc(top[2]) + __popc(top[3]);
    }
    // cost of k: k n + sum (q + 1), less one for each weight with q == qmax (its last plane is not closed)
    uint32_t best = 0xFFFFFFFFu, k_best = 0, qmax_best = 0, q_sum = 0;
#pragma unroll
    for (int b = 7; b >= 4; b--) q_sum = 2 * q_sum + sum[b];
    uint32_t cost[4];
#pragma unroll
    for (int k = 3; k >= 0; k--) {
      q_sum = 2 * q_sum + sum[k];
      cost[k] = k * n + q_sum + n - at_top[k];
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if ((rmax >> k) <= 63u && cost[k] < best) best = cost[k], k_best = k, qmax_best = rmax >> k;  // strict: ties keep the smaller k
    const int64_t row = task.row0 + sub;
    if (mine) meta[row * src.T + t] = (uint8_t)(k_best | (qmax_best << 2));
    const uint32_t upto = row_scan(mine ? best : 0u, lane, t, rows_per_task);
    if (rows_per_task > 1) {
      if (mine && t == src.T - 1) row_words[row] = (upto + 31) >> 5;
    } else {
      row_bits += __shfl_sync(BN_FULL, upto, 31);
      if (task.t0 + 32 >= src.T) {
        if (lane == 0) row_words[row] = (uint32_t)min((row_bits + 31) >> 5, (uint64_t)0xFFFFFFFFu);
        row_bits = 0;
      }
    }
  });
}

// roff = exclusive prefix sum of row_words (one block, 4096 rows a step, the next step's loads in
// flight); total[0] = number of words as uint64 (a total of 2^32 or more cannot be addressed by
// the format's uint32 offsets: the caller checks). 15360 rows: 21 us with 1024 rows a step.
__global__ void __launch_bounds__(1024) offsets_kernel(const uint32_t *__restrict__ row_words, int64_t R, uint32_t *__restrict__ roff, unsigned long long *__restrict__ total) {
  __shared__ unsigned long long warp_sum[2][32];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  unsigned long long carry = 0;
  auto load = [&](int64_t base, uint32_t (&v)[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int64_t i = base + threadIdx.x * 4 + j;
      v[j] = i < R ? row_words[i] : 0u;
    }
  };
  uint32_t v[4], next[4];
  load(0, next);
  int phase = 0;
  for (int64_t base = 0; base < R; base += 4096, phase ^= 1) {
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = next[j];
    if (base + 4096 < R) load(base + 4096, next);
    const unsigned long long own = (unsigned long long)v[0] + v[1] + v[2] + v[3];
    unsigned long long inc = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long n = __shfl_up_sync(BN_FULL, inc, d);
      if (lane >= (uint32_t)d) inc += n;
    }
    if (lane == 31) warp_sum[phase][warp] = inc;
    __syncthreads();  // (two copies of warp_sum: the next step's writes cannot meet this step's reads)
    unsigned long long before = warp_sum[phase][lane], all = before;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long n = __shfl_up_sync(BN_FULL, all, d);
      if (lane >= (uint32_t)d) all += n;
    }
    before = __shfl_sync(BN_FULL, all - before, warp);  // of the warps before this one
    const unsigned long long step_total = __shfl_sync(BN_FULL, all, 31);
    unsigned long long at = carry + before + inc - own;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int64_t i = base + threadIdx.x * 4 + j;
      if (i < R) roff[i] = (uint32_t)at;
      at += v[j];
    }
    carry += step_total;
  }
  if (threadIdx.x == 0) *total = carry;
}

// OR `n` <= 32 bits into the window at bit `pos` (counted from the window's first word)
__device__ __forceinline__ void put_bits(uint32_t *win, uint32_t pos, uint32_t v, uint32_t n) {
  if (!n) return;
  const uint32_t wi = pos >> 5, s = pos & 31u;
  atomicOr(win + wi, v << s);
  if (s + n > 32u) atomicOr(win + wi + 1, v >> (32u - s));
}
__global__ void __launch_bounds__(EN_WRITE_WARPS * 32, 1) write_kernel(EncSource src, const uint8_t *__restrict__ rank_table, const uint8_t *__restrict__ meta, const uint32_t *__restrict__ roff, int64_t R, int rows_per_task, uint32_t *__restrict__ bits, uint64_t nwords) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t *const pack = smem, *const rank = smem + EN_PACK, *const small = rank + 256;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t *const ranks = reinterpret_cast<uint32_t *>(smem + EN_PACK + 512) + warp * (EN_WORDS + EN_WINDOW), *const sh = ranks + EN_WORDS;
  if (threadIdx.x < 256) {
    rank[threadIdx.x] = rank_table[threadIdx.x];
    const uint32_t al = threadIdx.x >> 4, v = threadIdx.x & 15u;  // four bits: value | alive << 4
    uint32_t out = 0, c = 0;
    for (int i = 0; i < 4; i++)
      if ((al >> i) & 1u) out |= ((v >> i) & 1u) << c, c++;
    small[threadIdx.x] = (uint8_t)out;
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < EN_PACK / 4; e += EN_WRITE_WARPS * 32) {
    const uint32_t al = e >> 6, v = (e & 63u) * 4u, lo = (al & 15u) << 4, c = __popc(al & 15u);  // four values that differ in their lowest two bits
    const uint32_t up = (uint32_t)small[(v >> 4) | (al & 0xF0u)] << c;
    uint32_t word = 0;
    for (uint32_t i = 0; i < 4; i++) word |= (up | small[((v & 12u) + i) | lo]) << (8 * i);
    reinterpret_cast<uint32_t *>(pack)[e] = word;
  }
  __syncthreads();

  uint32_t row_at = 0;  // bits of the row before this chunk (one row a task)
  each_task(R, src.T, rows_per_task, warp, lane, [&](const EncTask &task, bool mine, int sub, int t) {
    uint32_t r[8][4];
    tile_planes(src, task, rank, ranks, lane, sub, t, r);
    const int64_t row = task.row0 + sub;
    const uint32_t m = mine ? meta[row * src.T + t] : 0u, k = m & 3u, qmax = m >> 2;
    const uint32_t n = mine ? (uint32_t)min((int64_t)BN_TILE, src.K - (int64_t)t * BN_TILE) : 0u;
    // the quotients' planes moved down: r[b] is bit b of q (r[6]: q has a bit above the third)
    uint32_t low[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      low[i] = r[0][i];
      uint32_t q[9];
#pragma unroll
      for (int b = 0; b < 8; b++) q[b] = r[b][i];
      q[8] = 0;
#pragma unroll
      for (int b = 0; b < 8; b++) q[b] = k & 1u ? q[b + 1] : q[b];
#pragma unroll
      for (int b = 0; b < 6; b++) q[b] = k & 2u ? q[b + 2] : q[b];
      // (q <= 63: six planes)
#pragma unroll
      for (int b = 0; b < 6; b++) r[b][i] = q[b];
      r[6][i] = q[3] | q[4] | q[5];
    }
    // the weights with q > j among those with q >= j, for the warp's plane j
    auto beyond = [&](const uint32_t (&alive)[4], uint32_t j, uint32_t (&next)[4]) {
      const uint32_t m0 = j & 1u ? 0u : 0xFFFFFFFFu, m1 = j & 2u ? 0u : 0xFFFFFFFFu, m2 = j & 4u ? 0u : 0xFFFFFFFFu;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        uint32_t same = (r[0][i] ^ m0) & (r[1][i] ^ m1) & (r[2][i] ^ m2);
        if (j < 8u) same &= ~r[6][i];
        else same &= (r[3][i] ^ (j & 8u ? 0u : 0xFFFFFFFFu)) & (r[4][i] ^ (j & 16u ? 0u : 0xFFFFFFFFu)) & (r[5][i] ^ (j & 32u ? 0u : 0xFFFFFFFFu));
        next[i] = alive[i] & ~same;
      }
    };
    // length: what the plan chose, counted again: k n, and per weight q + 1 planes, the last one of
    // qmax planes not closed
    uint32_t length = 0;
    if (mine) {
      uint32_t q_sum = 0, at_top[4];
#pragma unroll
      for (int b = 5; b >= 0; b--) q_sum = 2 * q_sum + __popc(r[b][0]) + __popc(r[b][1]) + __popc(r[b][2]) + __popc(r[b][3]);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        at_top[i] = low_mask((int)n - 32 * i);
#pragma unroll
        for (int b = 0; b < 6; b++) at_top[i] &= (qmax >> b) & 1u ? r[b][i] : ~r[b][i];
      }
      length = k * n + q_sum + n - (__popc(at_top[0]) + __popc(at_top[1]) + __popc(at_top[2]) + __popc(at_top[3]));
    }
    const uint32_t upto = row_scan(length, lane, t, rows_per_task);
    const uint32_t begin = row_at + upto - length, end = begin + length;  // bits of the row
    const uint64_t word0 = (uint64_t)roff[row] + (begin >> 5), word1 = (uint64_t)roff[row] + ((end + 31u) >> 5);  // words touched
    // (a tile without bits touches no word: word1 may be word0)
    for (int from = 0; from < task.count;) {
      // lanes from .. to - 1: those whose words fit the window together
      const uint64_t base = __shfl_sync(BN_FULL, word0, from);
      const bool fits = (int)lane == from || ((int)lane > from && mine && word0 >= base && word1 <= base + EN_WINDOW);
      const uint32_t gaps = ~(__ballot_sync(BN_FULL, fits) >> from);
      const int to = min(task.count, from + (gaps ? __ffs((int)gaps) - 1 : 32));
      const uint32_t words = (uint32_t)min(__shfl_sync(BN_FULL, max(word1, word0), to - 1) - base, (uint64_t)EN_WINDOW);
      // the window's first word may hold the last bits of what was written before
      const uint32_t carried = __shfl_sync(BN_FULL, begin & 31u, from) && base < nwords ? __ldcg(bits + base) : 0u;
      for (uint32_t i = lane; i < words; i += 32) sh[i] = i ? 0u : carried;
      __syncwarp();
      const bool active = (int)lane >= from && (int)lane < to;
      uint32_t pos = active ? (uint32_t)(word0 - base) * 32u + (begin & 31u) : 0u;
      uint32_t alive[4], next[4];
#pragma unroll
      for (int i = 0; i < 4; i++) alive[i] = active ? low_mask((int)n - 32 * i) : 0u;
      const uint8_t *const tile_ranks = reinterpret_cast<const uint8_t *>(ranks + lane * EN_TILE);
      if (active && k == 1) {  // low plane, one bit a weight: a bit plane as it is
#pragma unroll
        for (int i = 0; i < 4; i++) put_bits(sh, pos + 32 * i, low[i], max(0, min(32, (int)n - 32 * i)));
      } else if (active && k) {  // two or three bits a weight, out of the rank bytes
        const uint32_t km = (1u << k) - 1u;
        for (uint32_t i = 0; 4 * i < n; i++) {
          const uint32_t x = ranks[lane * EN_TILE + i];
          put_bits(sh, pos + 4 * i * k, (x & km) | ((x >> (8 - k)) & (km << k)) | ((x >> (16 - 2 * k)) & (km << (2 * k))) | ((x >> (24 - 3 * k)) & (km << (3 * k))), k * min(4u, n - 4 * i));
        }
      }
      pos += k * n;
      // unary planes
      uint32_t j = 0;
      for (;; j++) {
        if (j >= qmax) alive[0] = alive[1] = alive[2] = alive[3] = 0u;
        const uint32_t c0 = __popc(alive[0]), c1 = __popc(alive[1]), c2 = __popc(alive[2]), c3 = __popc(alive[3]), len = c0 + c1 + c2 + c3;
        if (__reduce_max_sync(BN_FULL, len) <= EN_FEW) break;
        beyond(alive, j, next);
        const uint32_t c[4] = {c0, c1, c2, c3};
#pragma unroll
        for (int i = 0; i < 4; i++) {
          uint32_t out = next[i];
          if (j) {  // (plane 0 has every weight)
            out = 0;
            uint32_t at = 0;
#pragma unroll
            for (int b = 0; b < 4; b++) {
              out |= (uint32_t)pack[__byte_perm(next[i], alive[i], 0x40 + 0x11 * b) & 0xFFFFu] << at;
              at += __popc(alive[i] & (0xFFu << (8 * b)));
            }
          }
          put_bits(sh, pos, out, c[i]);
          pos += c[i], alive[i] = next[i];
        }
      }
      // the few weights still alive, at most eight: their quotients in the bytes of q0 and q1
      uint32_t few, q0 = 0, q1 = 0, e = 0;
#pragma unroll
      for (int i = 0; i < 4; i++)
        for (uint32_t left = alive[i]; left; left &= left - 1u, e++) {
          const uint32_t q = (uint32_t)tile_ranks[32 * i + __ffs((int)left) - 1] >> k;
          if (e < 4u) q0 |= q << (8 * e);
          else q1 |= q << (8 * (e - 4u));
        }
      few = low_mask((int)e);
      for (; __any_sync(BN_FULL, few != 0); j++) {
        if (j >= qmax) few = 0;
        // bit 7 of a byte: q > j (both below 128)
        const uint32_t more0 = (q0 + (0x7Fu - j) * 0x01010101u) & 0x80808080u, more1 = (q1 + (0x7Fu - j) * 0x01010101u) & 0x80808080u;
        const uint32_t more = (((more0 >> 7) * 0x00204081u >> 21) & 15u) | (((more1 >> 7) * 0x00204081u >> 17) & 0xF0u);
        const uint32_t c = __popc(few);
        put_bits(sh, pos, pack[(more & few) | (few << 8)], c);
        pos += c, few &= more;
      }
      __syncwarp();
      for (uint32_t i = lane; i < words; i += 32)
        if (base + i < nwords) bits[base + i] = sh[i];  // never past the array
      __syncwarp();
      from = to;
    }
    row_at += rows_per_task > 1 ? 0u : __shfl_sync(BN_FULL, upto, 31);
    if (rows_per_task > 1 || task.t0 + 32 >= src.T) row_at = 0;
  });
}

// Grid and rows per task of the plan and the write: one block an SM.
struct EncShape {
  unsigned blocks;
  int rows_per_task;
};
EncShape enc_shape(int64_t R, int T) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // as many rows a task as keep every warp of the write at one task, up to the task's 32 tiles: tiles of
  // many planes fill the window six at a time, and a warp with 32 of them takes six turns while others
  // idle (random words, us: 64 x 128 144 -> 67, 1000 x 128 161 -> 69; ordinary words 72 -> 67)
  const int64_t all_warps = (int64_t)sms * EN_WRITE_WARPS;
  const int rows = T > 16 ? 1 : (int)max((int64_t)1, min((int64_t)(32 / T), (R + all_warps - 1) / all_warps));
  const int64_t tasks = (R + rows - 1) / rows;
  return {(unsigned)min(tasks, (int64_t)sms), rows};
}
EncSource enc_source(const uint16_t *w, int64_t K) {
  return {w, K, (int)tiles(K), K % 8 == 0 && !(reinterpret_cast<uintptr_t>(w) & 15)};
}

}  // namespace
}  // namespace bn

extern "C" int bn_bf16_split_hist(const uint16_t *w, int64_t n, uint8_t *raw, uint32_t *hist, void *stream) {
  if (!w || !raw || !hist || n < 0) return bn::fail(BN_ERR_ARG, "bn_bf16_split_hist: null pointer or negative size");
  cudaStream_t s = (cudaStream_t)stream;
  BN_CUDA(cudaMemsetAsync(hist, 0, 256 * sizeof(uint32_t), s));
  if (n == 0) return BN_OK;
  const int64_t per = bn::HIST_THREADS * 8, want = (n + per - 1) / per, blocks = want < 148 * 4 ? want : 148 * 4;
  const bool aligned = !((reinterpret_cast<uintptr_t>(w) & 15) | (reinterpret_cast<uintptr_t>(raw) & 7));
  bn::split_hist_kernel<<<(unsigned)blocks, bn::HIST_THREADS, 0, s>>>(w, n, raw, hist, aligned);
  return bn::launched("split_hist_kernel");
}

extern "C" int bn_rank_table(const uint32_t *hist, uint8_t *table, uint8_t *rank, void *stream) {
  if (!hist || !table || !rank) return bn::fail(BN_ERR_ARG, "bn_rank_table: null pointer");
  bn::rank_table_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(hist, table, rank);
  return bn::launched("rank_table_kernel");
}

extern "C" int bn_rice_encode_plan(const uint16_t *w, const uint8_t *rank, int64_t R, int64_t K, uint8_t *meta, uint32_t *row_words, uint32_t *roff, uint64_t *total, void *stream) {
  if (!w || !rank || !meta || !row_words || !roff || !total || R < 0 || K <= 0) return bn::fail(BN_ERR_ARG, "bn_rice_encode_plan: null pointer or bad size");
  cudaStream_t s = (cudaStream_t)stream;
  if (R == 0) {
    BN_CUDA(cudaMemsetAsync(total, 0, sizeof(uint64_t), s));
    return BN_OK;
  }
  const bn::EncSource src = bn::enc_source(w, K);
  const bn::EncShape shape = bn::enc_shape(R, src.T);
  constexpr size_t smem = 256 + bn::EN_WARPS * bn::EN_WORDS * 4;
  BN_CUDA(bn::allow_smem(bn::plan_kernel, smem));
  bn::plan_kernel<<<shape.blocks, bn::EN_WARPS * 32, smem, s>>>(src, rank, R, shape.rows_per_task, meta, row_words);
  if (int e = bn::launched("plan_kernel")) return e;
  bn::offsets_kernel<<<1, 1024, 0, s>>>(row_words, R, roff, reinterpret_cast<unsigned long long *>(total));
  return bn::launched("offsets_kernel");
}

extern "C" int bn_rice_encode_write(const uint16_t *w, const uint8_t *rank, const uint8_t *meta, const uint32_t *roff, int64_t R, int64_t K, uint32_t *bits, uint64_t nwords, void *stream) {
  if (!w || !rank || !meta || !roff || (!bits && nwords) || R < 0 || K <= 0) return bn::fail(BN_ERR_ARG, "bn_rice_encode_write: null pointer or bad size");
  if (R == 0) return BN_OK;
  const bn::EncSource src = bn::enc_source(w, K);
  const bn::EncShape shape = bn::enc_shape(R, src.T);
  BN_CUDA(bn::allow_smem(bn::write_kernel, bn::EN_SMEM));
  bn::write_kernel<<<shape.blocks, bn::EN_WRITE_WARPS * 32, bn::EN_SMEM, (cudaStream_t)stream>>>(src, rank, meta, roff, R, shape.rows_per_task, bits, nwords);
  return bn::launched("write_kernel");
}
