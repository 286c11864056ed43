// Format-2 (Rice) stream decode, one thread per tile.
//
// A tile's length is only known once its planes are counted, but counting is cheap: plane j + 1
// has as many bits as plane j has ones. So the chain over a row's tiles is taken out of the decode:
//
//   rice_scan_kernel   a thread per row walks the row by population counts and writes every tile's
//                      first bit; the stream comes through a ring in shared memory
//   rice_tiles_kernel  a thread per tile: alive masks are four 32-bit words, the bits of a plane
//                      are deposited on the alive positions eight weights at a time through a
//                      table in shared memory, quotients are counted in bit planes, and the four
//                      bit planes of min(rank, 15) are transposed to nibbles in registers
//
// The decoder with a warp per row (rice_kernel) spends a warp-wide step on every plane of every
// tile, 240 to 500 warp instructions a tile; here 30 tiles share 2470, and the scan adds 52 a tile.
// Measured with the benchmark's distribution (us, warp per row -> here): R4 arrays of 15360 x 3840
// 192 -> 41 + 63 (scan + tiles), of 3840 x 15360 350 -> 113 + 72; BF16 words of 22528 x 704 97 -> 12 + 36.
// Escapes cost little while they are few: a tile's last eight weights are at hand, the others come out
// of one more walk over its planes, and tiles with three low bits, where most weights escape, are
// decoded one at a time by the whole warp (rice_kernels.cu takes streams that are full of such tiles).
// The tiles' first bits wait in the output array itself (the last 4 T bytes of each output row):
// entry t lies in the bytes of tile t or later, and a row's tiles are decoded in order by one
// warp that reads its entries first, so no entry is overwritten before it is read.
#include "rice.cuh"

namespace bn {
namespace {

// ---------------------------------------------------------------------------------------------
// First bits of the tiles
// ---------------------------------------------------------------------------------------------
constexpr uint32_t SC_BLOCK = 128;                   // words of a ring block
constexpr uint32_t SC_RING = 2 * SC_BLOCK;           // words of a row's ring
constexpr uint32_t SC_STRIDE = SC_RING + 12;         // the ring's first 12 words again at its end: a read of up to 12 words never wraps

// Words from nwords on read as zero.
__device__ __forceinline__ uint32_t word_at(const uint32_t *__restrict__ bits, uint64_t nwords, uint64_t i) { return i < nwords ? __ldg(bits + i) : 0u; }
// First word of a row in `bits` (an offset past every stream stays one).
__device__ __forceinline__ uint32_t row_word(const RiceArgs &a, int64_t row) { return min(a.roff[row], 0xFFFFFFFFu - a.shift) + a.shift; }
// (hi:lo) >> n, n <= 32
__device__ __forceinline__ void shift_out(uint32_t &lo, uint32_t &hi, uint32_t n) {
  lo = __funnelshift_rc(lo, hi, n);
  asm("shr.b32 %0, %0, %1;" : "+r"(hi) : "r"(n));
}

// Bit after the tile that starts at bit `cur` of the row's ring space, for tiles that might not fit the
// ring: words before `limit` come from there, the others from global memory (`row` is where the
// ring space starts). The four lanes of a row count 32 bits of a plane each.
__device__ __noinline__ uint32_t scan_long_tile(const uint32_t *__restrict__ bits, uint64_t nwords, uint64_t row, uint32_t ring, uint32_t limit, uint32_t cur, uint32_t n, uint32_t k, uint32_t qmax) {
  const uint32_t lane = lane_id(), mask = 15u << (lane & 28u);
  auto word = [&](uint32_t w) { return w < limit ? lds_u32(ring + 4u * (w & (SC_RING - 1u))) : word_at(bits, nwords, row + w); };
  uint32_t pos = cur + n * k, len = n, j = 0;
  for (; j < qmax && len > 32u; j++) {
    const uint32_t at = pos + 32u * (lane & 3u), w = at >> 5;
    uint32_t ones = __popc(__funnelshift_r(word(w), word(w + 1u), at & 31u) & low_mask((int)(len - 32u * (lane & 3u))));
    ones += __shfl_xor_sync(mask, ones, 1);
    ones += __shfl_xor_sync(mask, ones, 2);
    pos += len, len = ones;
  }
  uint32_t lo = 0, hi = 0, room = 0;  // a window of the bits from pos on
  for (; j < qmax && len; j++) {
    if (len > room) {
      const uint32_t w = pos >> 5, v = word(w + 1u);
      lo = __funnelshift_r(word(w), v, pos & 31u), hi = __funnelshift_r(v, word(w + 2u), pos & 31u), room = 64;
    }
    const uint32_t ones = __popc(lo & low_mask((int)len));
    shift_out(lo, hi, len);
    pos += len, room -= len, len = ones;
  }
  return pos;
}

// One warp per block, four lanes per row (`rows_per_block` <= 8 rows): a lane counts 32 of up to 128
// bits of a plane; planes of few bits are counted by all four alike. slots + (row + 1) * row_bytes -
// 4 (T - t) receives tile t's first bit, counted from the row's first word.
// Bound: the instructions of a row's chain of dependent counts (366 a step, 57 % of issue slots).
// With a row per lane the walk takes 537 instructions a step (the slowest of 26 rows decides each
// loop) in a quarter of the warps: as long on 15360 rows (44 us), longer on fewer.
template <int MODE>
__global__ void __launch_bounds__(32) rice_scan_kernel(RiceArgs a, uint8_t *slots, int64_t row_bytes, int rows_per_block) {
  extern __shared__ __align__(16) uint32_t ring_all[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the decode's blocks build their tables meanwhile
  const uint32_t lane = lane_id(), part = lane & 3u;
  const int64_t row = (int64_t)blockIdx.x * rows_per_block + (lane >> 2);
  bool live = (int)(lane >> 2) < rows_per_block && row < a.R;
  const int T = a.T;
  int64_t srow = live ? row : 0;
  if (MODE == RICE_UNPACK && a.ids) {
    srow = live ? (int64_t)a.ids[row] : 0;
    if (srow >= a.rows) live = false, srow = 0;  // an id outside the table: the decode writes zeros
  }
  const uint32_t w0 = live ? row_word(a, srow) : 0u;
  const uint32_t first = w0 & ~3u;  // the ring starts at a 16-byte boundary of the stream
  const uint32_t avail = (uint64_t)first < a.nwords ? (uint32_t)min(a.nwords - first, (uint64_t)0xFFFFFFFFu) : 0u;
  const uint32_t off = (w0 & 3u) * 32u;
  const uint8_t *const meta = a.meta + srow * T;
  uint32_t *const slot = reinterpret_cast<uint32_t *>(slots + (row + 1) * row_bytes) - T;
  const uint32_t *const ring = ring_all + min(lane >> 2, (uint32_t)rows_per_block - 1u) * SC_STRIDE;
  int t = live ? 0 : T;
  uint32_t cur = off, req = 0, usable = 0;  // bit of the row's ring space; ring blocks asked for; blocks that have landed
  uint32_t m_next = live ? meta[0] : 0u;
  uint32_t bound = 0;
  for (;;) {
    // ask for the blocks up to the one after the cursor's
    for (;;) {
      req = max(req, cur >> 12);
      uint32_t want = __ballot_sync(BN_FULL, part == 0 && t < T && req < (cur >> 12) + 2u);
      if (!want) break;
      while (want) {
        const int i = __ffs((int)want) - 1;
        want &= want - 1u;
        const uint32_t b = __shfl_sync(BN_FULL, req, i), f = __shfl_sync(BN_FULL, first, i), av = __shfl_sync(BN_FULL, avail, i);
        const uint32_t w = b * SC_BLOCK + lane * 4u;
        const uint32_t bytes = w < av ? min(av - w, 4u) * 4u : 0u;  // past the stream: zeros
        const uint32_t *src = bytes ? a.bits + f + w : a.bits;
        const uint32_t dst = smem_addr(ring_all + (uint32_t)(i >> 2) * SC_STRIDE + (b & 1u) * SC_BLOCK + lane * 4u);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
        if ((b & 1u) == 0 && lane < 3) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + SC_RING * 4u), "l"(src), "r"(bytes) : "memory");
        if ((lane >> 2) == (uint32_t)(i >> 2)) req++;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // walk tiles while they lie in blocks that have landed; the loops below are the warp's
    for (;;) {
      const uint32_t m = m_next, k = m & 3u, qmax = m >> 2;
      const uint32_t n = (uint32_t)min((int64_t)BN_TILE, a.K - (int64_t)t * BN_TILE);
      const uint32_t most = n * (k + qmax);
      const bool is_long = most > SC_BLOCK * 32u;
      const bool go = t < T && cur + min(most, SC_BLOCK * 32u) <= usable * (SC_BLOCK * 32u);  // (a long tile starts with a block's length of bits at hand)
      if (!__any_sync(BN_FULL, go)) break;
      if (go) {
        if (part == 0) slot[t] = cur - off;
        if (t + 1 < T) m_next = meta[t + 1];
        if (MODE == RICE_R4 && part == 0 && ((qmax << k) | ((1u << k) - 1u)) >= 15u) bound += n;  // only such a tile can hold a rank >= 15
        if (is_long) cur = scan_long_tile(a.bits, a.nwords, first, smem_addr(ring), usable * SC_BLOCK, cur, n, k, qmax);
        t++;
      }
      const uint32_t planes = go && !is_long ? qmax : 0u;
      uint32_t pos = cur + n * k, len = n, j = 0;
      for (;;) {
        const bool act = j < planes && len > 32u;
        if (!__any_sync(BN_FULL, act)) break;
        const uint32_t at = pos + 32u * part;
        const uint32_t *p = ring + ((at >> 5) & (SC_RING - 1u));
        uint32_t ones = __popc(__funnelshift_r(p[0], p[1], at & 31u) & low_mask((int)(len - 32u * part)));
        ones += __shfl_xor_sync(BN_FULL, ones, 1);
        ones += __shfl_xor_sync(BN_FULL, ones, 2);
        if (act) pos += len, len = ones, j++;
      }
      uint32_t lo = 0, hi = 0, room = 0;  // a window of the bits from pos on
      auto refill = [&]() {
        const uint32_t *p = ring + ((pos >> 5) & (SC_RING - 1u));
        const uint32_t sh = pos & 31u, v1 = p[1];
        lo = __funnelshift_r(p[0], v1, sh), hi = __funnelshift_r(v1, p[2], sh), room = 64;
      };
      while (j < planes && len > 1u) {
        if (len > room) refill();
        const uint32_t ones = __popc(lo & low_mask((int)len));
        shift_out(lo, hi, len);
        pos += len, room -= len, len = ones, j++;
      }
      if (j < planes && len) {  // the last weight's planes are a run of ones closed by a zero, or by reaching qmax
        refill();
        const uint32_t rem = planes - j, low = (uint32_t)__clz((int)__brev(~lo)), run = low < 32u ? low : 32u + (uint32_t)__clz((int)__brev(~hi));
        pos += min(run + 1u, rem);
      }
      if (go && !is_long) cur = pos;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    usable = req;
    if (!__any_sync(BN_FULL, t < T)) break;
  }
  const uint32_t rend = w0 - a.shift + ((cur - off + 31u) >> 5);
  if (MODE == RICE_R4) {
    // escape scratch for the most escapes the rows' meta bytes allow, claimed once per warp
    uint32_t upto = bound;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(BN_FULL, upto, d);
      if (lane >= (uint32_t)d) upto += v;
    }
    uint32_t claim = 0;
    if (lane == 31 && upto) claim = (uint32_t)atomicAdd(reinterpret_cast<unsigned long long *>(a.counters + 4), (unsigned long long)upto);
    claim = __shfl_sync(BN_FULL, claim, 31);
    if (!live || part) return;
    a.tmp_off[row] = claim + upto - bound;
    const uint64_t w_end = row + 1 < a.R ? (uint64_t)a.roff[row + 1] : a.nwords - a.shift;
    if ((uint64_t)rend != w_end) atomicMax(a.counters + 1, (uint32_t)(a.R - row));
  } else if (live && part == 0 && a.rend) {
    a.rend[row] = rend;
  }
}

// ---------------------------------------------------------------------------------------------
// The tiles
// ---------------------------------------------------------------------------------------------
constexpr int TI_WARPS = 28;
constexpr uint32_t TI_WORDS = 512;                  // stream words a warp stages at a time (a tile has at most 265)
constexpr uint32_t TI_TILE = 20;                    // words between two tiles' codes in shared memory: 16, and no bank conflicts for 16-byte accesses
constexpr uint32_t TI_DEPOSIT = 65536;              // byte [bits | alive << 8]: the low bits of `bits`, in order, on the set positions of `alive`
constexpr uint32_t TI_WARP_WORDS = TI_WORDS + 12 + 32 * TI_TILE;
constexpr uint32_t TI_SMEM = TI_DEPOSIT + 1024 + 256 + 256 + TI_WARPS * TI_WARP_WORDS * 4;
constexpr uint32_t TI_FEW = 8;                      // alive weights up to which a tile is finished as one deposit of eight bits a plane

__device__ __forceinline__ uint32_t window(const uint32_t *sw, uint32_t pos) {
  const uint32_t *p = sw + (pos >> 5);
  return __funnelshift_r(p[0], p[1], pos & 31u);
}
// Bits 2m of x packed together (16 of them).
__device__ __forceinline__ uint32_t pack2(uint32_t x) {
  x &= 0x55555555u;
  x = (x | (x >> 1)) & 0x33333333u;
  x = (x | (x >> 2)) & 0x0F0F0F0Fu;
  x = (x | (x >> 4)) & 0x00FF00FFu;
  return (x | (x >> 8)) & 0xFFFFu;
}
// Bit planes r0..r3 of 32 nibbles -> the nibbles, eight a word, in order.
__device__ __forceinline__ uint4 nibbles(uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  uint32_t t;
  auto swap = [&](uint32_t &x, uint32_t &y, int sh, uint32_t mask) { t = ((x >> sh) ^ y) & mask, y ^= t, x ^= t << sh; };
  swap(r0, r1, 1, 0x55555555u), swap(r2, r3, 1, 0x55555555u);  // pairs of bits of weights 2m (r0, r2) and 2m + 1 (r1, r3)
  swap(r0, r2, 2, 0x33333333u), swap(r1, r3, 2, 0x33333333u);  // nibbles of weights 4g (r0), 4g + 1 (r1), 4g + 2 (r2), 4g + 3 (r3)
  swap(r0, r1, 4, 0x0F0F0F0Fu), swap(r2, r3, 4, 0x0F0F0F0Fu);  // bytes of weights 8i, 8i + 1 (r0), 8i + 4, 5 (r1), 8i + 2, 3 (r2), 8i + 6, 7 (r3)
  const uint32_t a01 = __byte_perm(r0, r2, 0x5140), a23 = __byte_perm(r0, r2, 0x7362), b01 = __byte_perm(r1, r3, 0x5140), b23 = __byte_perm(r1, r3, 0x7362);
  return make_uint4(__byte_perm(a01, b01, 0x5410), __byte_perm(a01, b01, 0x7632), __byte_perm(a23, b23, 0x5410), __byte_perm(a23, b23, 0x7632));
}

// A warp takes `rows_per_task` whole rows (several when 32 tiles hold them), 32 tiles at a time.
// Bound: shared memory (61 % of its cycles: the deposit table's conflicts) and issue (63 %). Of the
// 2470 instructions of a 30-tile row a plane's deposits take 164, about five planes of them; with
// the last few weights of a plane taken one by one instead of as one more deposit the kernel took
// 95 us on 15360 x 3840.
template <int MODE>
__global__ void __launch_bounds__(TI_WARPS * 32, 1) rice_tiles_kernel(RiceArgs a, const uint8_t *slots, int64_t row_bytes, int rows_per_task) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t *const deposit = smem;
  uint32_t *const pair = reinterpret_cast<uint32_t *>(smem + TI_DEPOSIT);  // two codes -> their exponents in a BF16x2 word; code 15: none
  uint8_t *const tbl = smem + TI_DEPOSIT + 1024;
  uint8_t *const small = tbl + 256;  // the deposit of four bits: alive | bits << 4
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t *const sw = reinterpret_cast<uint32_t *>(smem + TI_DEPOSIT + 1536) + warp * TI_WARP_WORDS;
  uint32_t *const sc = sw + TI_WORDS + 12;
  if (threadIdx.x < 256) {
    const uint32_t al = threadIdx.x & 15u;
    uint32_t b = threadIdx.x >> 4, out = 0;
    for (int i = 0; i < 4; i++)
      if ((al >> i) & 1u) out |= (b & 1u) << i, b >>= 1;
    small[threadIdx.x] = (uint8_t)out;
    tbl[threadIdx.x] = a.table[threadIdx.x];
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < TI_DEPOSIT / 4; e += TI_WARPS * 32) {  // four values of the bits' lowest two at once
    const uint32_t al = e >> 6, b = e & 63u, p0 = al & (0u - al), rest = al ^ p0, p1 = rest & (0u - rest), up = rest ^ p1, c = __popc(up & 15u);
    const uint32_t base = small[(up & 15u) | ((b & 15u) << 4)] | ((uint32_t)small[(up >> 4) | (((b >> c) & 15u) << 4)] << 4);
    reinterpret_cast<uint32_t *>(deposit)[e] = base * 0x01010101u | (p0 << 8) | (p1 << 16) | ((p0 | p1) << 24);
  }
  if (MODE == RICE_UNPACK && threadIdx.x < 256) {
    const uint32_t c0 = threadIdx.x & 15u, c1 = threadIdx.x >> 4;
    pair[threadIdx.x] = (c0 == 15u ? 0u : (uint32_t)tbl[c0] << 7) | (c1 == 15u ? 0u : (uint32_t)tbl[c1] << 23);
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the tiles' first bits

  const int T = a.T;
  const bool quads = !(reinterpret_cast<uintptr_t>(a.codes) & 15);  // (8-byte aligned else)
  const int64_t K = a.K, tasks = (a.R + rows_per_task - 1) / rows_per_task;
  uint32_t escapes = 0;  // of the rows whose count this lane stores
  for (int64_t task = (int64_t)warp * gridDim.x + blockIdx.x; task < tasks; task += (int64_t)gridDim.x * TI_WARPS) {
    const int64_t row0 = task * rows_per_task;
    const int rows = (int)min((int64_t)rows_per_task, a.R - row0);
    if (MODE == RICE_UNPACK && a.ids && (int64_t)a.ids[row0] >= a.rows) {  // an id outside the table: a row of zeros
      for (int64_t c = lane; c < K / 4; c += 32) *reinterpret_cast<uint2 *>(a.out + row0 * K + c * 4) = make_uint2(0, 0);
      continue;
    }
    uint32_t row_escapes = 0;  // of the tiles before this chunk (one row a task)
    for (int t0 = 0; t0 < T; t0 += 32) {
      // this lane's tile
      const int tiles_here = rows > 1 ? rows * T : min(32, T - t0);
      const bool mine = (int)lane < tiles_here;
      const int sub = rows_per_task > 1 ? (int)lane / T : 0, t = mine ? (rows_per_task > 1 ? (int)lane - sub * T : t0 + (int)lane) : 0;
      const int64_t row = row0 + (mine ? sub : 0);
      const int64_t srow = MODE == RICE_UNPACK && a.ids ? (int64_t)a.ids[row] : row;
      const uint32_t m = a.meta[srow * T + t], k = m & 3u, qmax = m >> 2;
      const uint32_t n = (uint32_t)min((int64_t)BN_TILE, K - (int64_t)t * BN_TILE);
      const uint32_t *const slot = reinterpret_cast<const uint32_t *>(slots + (row + 1) * row_bytes) - T;
      const uint32_t w0 = row_word(a, srow), begin = slot[t], end = t + 1 < T ? slot[t + 1] : begin + n * (k + qmax);
      const uint32_t first_word = w0 + (begin >> 5), last_word = w0 + (end >> 5);
      // the raw bytes are only needed once the tiles are decoded: on their way to L2 meanwhile
      if (MODE == RICE_UNPACK && mine) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.raw + srow * K + (int64_t)t * BN_TILE));
      __syncwarp();  // every entry of the chunk is read before anything is written
      uint32_t hits[4] = {0, 0, 0, 0}, low_at = 0, planes_at = 0, count = 0;
      for (int from = 0; from < tiles_here;) {
        // lanes from .. to - 1: those whose tiles fit the staged words together
        const uint32_t base = __shfl_sync(BN_FULL, first_word, from) & ~3u;  // a 16-byte boundary of the stream
        const bool fits = (int)lane == from || ((int)lane > from && mine && first_word >= base && last_word - base < TI_WORDS);
        const uint32_t gaps = ~(__ballot_sync(BN_FULL, fits) >> from);
        const int to = min(tiles_here, from + (gaps ? __ffs((int)gaps) - 1 : 32));
        const uint32_t words = min(__shfl_sync(BN_FULL, last_word, to - 1) - base + 1u, TI_WORDS) + 8u;
        __syncwarp();
        if ((uint64_t)base + words + 3u <= a.nwords) {
          const uint4 *const src = reinterpret_cast<const uint4 *>(a.bits + base);
          for (uint32_t i = lane; i < (words + 3u) / 4u; i += 32) *reinterpret_cast<uint4 *>(sw + i * 4u) = __ldg(src + i);
        } else {
          for (uint32_t i = lane; i < words; i += 32) sw[i] = word_at(a.bits, a.nwords, (uint64_t)base + i);
        }
        __syncwarp();
        const bool active = (int)lane >= from && (int)lane < to;
        if (active) low_at = (first_word - base) * 32u + (begin & 31u), planes_at = low_at + n * k;
        const uint32_t shared_tiles = __ballot_sync(BN_FULL, active && k == 3);  // the warp decodes each together
        const bool own = active && k < 3;
        uint32_t alive[4], q0[4], q1[4], q2[4], q3[4], sat[4];
        const uint32_t q_top = 15u >> k;  // quotients above it mean rank >= 15
        uint32_t pos = own ? planes_at : 0u;
        const bool coded = own && qmax > 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          alive[i] = coded ? window(sw, pos + 32 * i) & low_mask((int)n - 32 * i) : 0u;  // plane 0
          q0[i] = alive[i], q1[i] = q2[i] = q3[i] = sat[i] = 0u;
        }
        if (coded) pos += n;
        // one more for the survivors of plane j (which holds j + 1 for them now)
        auto bump = [&](uint32_t j) {
          if (j >= q_top) {
#pragma unroll
            for (int i = 0; i < 4; i++) sat[i] |= alive[i];
          } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
              q0[i] ^= alive[i];
              if (j & 1u) q1[i] ^= alive[i];
              if ((j & 3u) == 3u) q2[i] ^= alive[i];
              if ((j & 7u) == 7u) q3[i] ^= alive[i];
            }
          }
        };
        uint32_t j = 1;
        for (;; j++) {
          if (j >= qmax) alive[0] = alive[1] = alive[2] = alive[3] = 0u;  // alive after the last plane: q = qmax
          const uint32_t c0 = __popc(alive[0]), c1 = __popc(alive[1]), c2 = __popc(alive[2]), c3 = __popc(alive[3]), len = c0 + c1 + c2 + c3;
          const uint32_t longest = __reduce_max_sync(BN_FULL, len);
          if (longest > TI_FEW) {
            const uint32_t at[4] = {pos, pos + c0, pos + c0 + c1, pos + c0 + c1 + c2};
#pragma unroll
            for (int i = 0; i < 4; i++) {
              uint32_t bits = window(sw, at[i]), next = 0;
#pragma unroll
              for (int b = 0; b < 4; b++) {
                const uint32_t d = deposit[__byte_perm(bits, alive[i], 0x40 + 0x10 * b) & 0xFFFFu];
                bits >>= __popc(alive[i] & (0xFFu << (8 * b)));
                next |= d << (8 * b);
              }
              alive[i] = next;
            }
            pos += len;
          } else {
            break;
          }
          bump(j);
        }
        // the few weights still alive, at most eight: one bit each of `few`, their further planes
        // counted in the bytes of more0 and more1 (a byte holds 63 at most)
        uint32_t few = 0, more0 = 0, more1 = 0;
        {
          const uint32_t len = __popc(alive[0]) + __popc(alive[1]) + __popc(alive[2]) + __popc(alive[3]);
          few = low_mask((int)len);
          for (uint32_t i = j; __any_sync(BN_FULL, few != 0); i++) {
            if (i >= qmax) few = 0;
            const uint32_t bits = window(sw, pos);
            pos += __popc(few);
            few = deposit[__byte_perm(bits, few, 0x40) & 0xFFFFu];
            more0 += ((few & 15u) * 0x00204081u) & 0x01010101u, more1 += ((few >> 4) * 0x00204081u) & 0x01010101u;
          }
        }
        // the low bits as bit planes under the quotients'
        if (own) {
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const uint32_t valid = low_mask((int)n - 32 * i);
            uint32_t r0 = q0[i], r1 = q1[i], r2 = q2[i], r3 = q3[i];
            if (k) {
              r3 = r2, r2 = r1, r1 = r0;
              if (k == 1) {
                r0 = window(sw, low_at + 32 * i) & valid;
              } else {
                r3 = r2, r2 = r1;
                const uint32_t x = valid ? window(sw, low_at + 64 * i) : 0u, y = valid & 0xFFFF0000u ? window(sw, low_at + 64 * i + 32) : 0u;
                r0 = (pack2(x) | (pack2(y) << 16)) & valid, r1 = (pack2(x >> 1) | (pack2(y >> 1) << 16)) & valid;
              }
            }
            r0 |= sat[i], r1 |= sat[i], r2 |= sat[i], r3 |= sat[i];
            hits[i] = r0 & r1 & r2 & r3;
            *reinterpret_cast<uint4 *>(sc + lane * TI_TILE + 4 * i) = nibbles(r0, r1, r2, r3);
          }
          // the further planes of the few, added to their nibbles
          uint32_t c = 0;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            for (uint32_t left = more0 | more1 ? alive[i] : 0u; left; left &= left - 1u, c++) {
              const uint32_t more = __byte_perm(more0, more1, 0x4440u | c) & 0xFFu;
              if (!more) continue;
              const uint32_t at = (uint32_t)__ffs((int)left) - 1u, sh = (at & 7u) * 4u;
              uint32_t *const word = sc + lane * TI_TILE + 4 * i + (at >> 3);
              const uint32_t old = (*word >> sh) & 15u, now = min(old + (more << k), 15u);
              *word += (now - old) << sh;
              if (now == 15u) hits[i] |= left & (0u - left);
            }
          }
          count = __popc(hits[0]) + __popc(hits[1]) + __popc(hits[2]) + __popc(hits[3]);
        }
        // exponents of the escaped weights (rank >= 15) with their place among the tile's: of the few
        // by their counts; the others' quotients are where they die in one more walk over the
        // planes, which such a tile alone takes
        auto each_escape = [&](auto &&put) {
          uint32_t c = 0, hits_before[4], left[4];
#pragma unroll
          for (int i = 0; i < 4; i++) hits_before[i] = c, c += __popc(hits[i]), left[i] = hits[i] & ~alive[i];
          auto place = [&](int i, uint32_t bit, uint32_t q) {
            const uint32_t at = 32u * i + (uint32_t)__ffs((int)bit) - 1u;
            put(at, (uint32_t)tbl[((q << k) | (k ? window(sw, low_at + at * k) & ((1u << k) - 1u) : 0u)) & 0xFFu], hits_before[i] + __popc(hits[i] & (bit - 1u)));
          };
          c = 0;  // of the few: those before this word
#pragma unroll
          for (int i = 0; i < 4; i++) {
            for (uint32_t h = hits[i] & alive[i]; h; h &= h - 1u) {
              const uint32_t bit = h & (0u - h);
              place(i, bit, j + (__byte_perm(more0, more1, 0x4440u | (c + __popc(alive[i] & (bit - 1u)))) & 0xFFu));
            }
            c += __popc(alive[i]);
          }
          uint32_t live[4], at = planes_at;
#pragma unroll
          for (int i = 0; i < 4; i++) live[i] = low_mask((int)n - 32 * i);
          for (uint32_t q = 0; left[0] | left[1] | left[2] | left[3]; q++) {  // (alive after the last plane: q = qmax)
#pragma unroll
            for (int i = 0; i < 4; i++) {
              uint32_t bits = window(sw, at), next = 0;
              at += __popc(live[i]);
#pragma unroll
              for (int b = 0; b < 4; b++) {
                next |= (uint32_t)deposit[__byte_perm(bits, live[i], 0x40 + 0x10 * b) & 0xFFFFu] << (8 * b);
                bits >>= __popc(live[i] & (0xFFu << (8 * b)));
              }
              if (q >= qmax) next = 0;
              for (uint32_t h = left[i] & ~next; h; h &= h - 1u) place(i, h & (0u - h), q);
              live[i] = next, left[i] &= next;
            }
          }
        };
        // tiles with k = 3, one after the other: four weights a lane, their ranks in the bytes of a word
        auto each_shared = [&](auto &&take) {
          for (uint32_t rest = shared_tiles; rest; rest &= rest - 1u) {
            const int u = __ffs((int)rest) - 1;
            const uint32_t un = __shfl_sync(BN_FULL, n, u), planes = __shfl_sync(BN_FULL, qmax, u), low = __shfl_sync(BN_FULL, low_at, u);
            const uint32_t nv = (uint32_t)max(0, min(4, (int)un - 4 * (int)lane));
            uint32_t four = (1u << nv) - 1u, q = 0, at = low + 3u * un;
            for (uint32_t plane = 0; plane < planes; plane++) {
              const uint32_t c = __popc(four);
              uint32_t before, all;
              warp_scan_small(c, lanemask_lt(), before, all);
              if (!all) break;
              four = small[four | ((window(sw, at + before) & low_mask((int)c)) << 4)];  // the survivors
              q += (four * 0x00204081u) & 0x01010101u;
              at += all;
            }
            const uint32_t x = nv ? window(sw, low + 12u * lane) : 0u;
            const uint32_t lows = (x & 7u) | ((x << 5) & 0x700u) | ((x << 10) & 0x70000u) | ((x << 15) & 0x7000000u);
            take(u, nv, (((q & 0x1F1F1F1Fu) << 3) | lows) & low_mask((int)(8u * nv)));
          }
        };
        __syncwarp();
        if (MODE == RICE_R4) {
          const uint64_t esc_at = (uint64_t)a.tmp_off[row] + (rows_per_task > 1 ? __shfl_sync(BN_FULL, row_escapes, mine ? sub * T : 0) : row_escapes);  // of this lane's row, the chunk's earlier ones included
          each_shared([&](int u, uint32_t, uint32_t ranks) {
            const uint32_t over = (((ranks & 0x7F7F7F7Fu) + 0x71717171u) | ranks) & 0x80808080u;  // bit 7 of the bytes from 15 on
            uint32_t c = (ranks | ((over >> 7) * 15u)) & 0x0F0F0F0Fu;
            c = (c | (c >> 4)) & 0x00FF00FFu;
            reinterpret_cast<uint16_t *>(sc + u * TI_TILE)[lane] = (uint16_t)(c | (c >> 8));
            const int usub = __shfl_sync(BN_FULL, sub, u);
            const uint32_t earlier = __reduce_add_sync(BN_FULL, (int)lane < u && sub == usub && active ? count : 0u);
            uint32_t before, all;
            warp_scan_small(__popc(over), lanemask_lt(), before, all);
            uint64_t p = __shfl_sync(BN_FULL, esc_at, u) + earlier + before;
#pragma unroll
            for (int i = 0; i < 4; i++)
              if ((over >> (8 * i + 7)) & 1u) {
                if (p < a.esc_cap) a.esc_tmp[p] = tbl[(ranks >> (8 * i)) & 0xFFu];
                p++;
              }
            if ((int)lane == u) count = all;
          });
          __syncwarp();
          const int64_t tile0 = row0 * T + t0 + from;  // the chunk's tiles are consecutive in memory
          uint4 *const dst = reinterpret_cast<uint4 *>(a.codes + tile0 * 32);
          for (int i = (int)lane; i < (to - from) * 4; i += 32) {
            const uint4 v = *reinterpret_cast<const uint4 *>(sc + (from + (i >> 2)) * TI_TILE + (i & 3) * 4);
            if (quads) dst[i] = v;
            else reinterpret_cast<uint2 *>(dst + i)[0] = make_uint2(v.x, v.y), reinterpret_cast<uint2 *>(dst + i)[1] = make_uint2(v.z, v.w);
          }
          if (active) a.flags[row0 * T + t0 + lane] = count != 0;
          if (!active) count = 0;
          if (__any_sync(BN_FULL, count != 0)) {
            uint32_t upto = count;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
              const uint32_t v = __shfl_up_sync(BN_FULL, upto, d);
              if (lane >= (uint32_t)d) upto += v;
            }
            const uint32_t total = __shfl_sync(BN_FULL, upto, 31);
            // several rows a task: positions count from the row's first tile
            const uint32_t before = __shfl_sync(BN_FULL, upto - count, rows_per_task > 1 ? max(sub * T, from) & 31 : 0);
            const uint64_t p = esc_at + (upto - count) - (rows_per_task > 1 ? before : 0u);
            if (own && count) each_escape([&](uint32_t, uint32_t e, uint32_t index) {
              if (p + index < a.esc_cap) a.esc_tmp[p + index] = (uint8_t)e;
            });
            if (rows_per_task == 1) {
              row_escapes += total;
            } else {  // each row's own count, kept by its first lane
              const int last = mine ? min(sub * T + T, 32) - 1 : 0;
              const uint32_t to_end = __shfl_sync(BN_FULL, upto, last);
              row_escapes += mine ? to_end - before : 0u;
            }
          }
        } else {
          // BF16 words: eight lanes a tile, sixteen weights a lane
          const bool wide = (K & 15) == 0;
          // the raw bytes of step u0 (four tiles), one step ahead of their use
          struct Piece {
            int64_t row, col;
            uint32_t rw[4];
          };
          auto fetch = [&](int u0) {
            const int u = u0 + (int)(lane >> 3);
            const int us = __shfl_sync(BN_FULL, sub, u & 31), ut = __shfl_sync(BN_FULL, t, u & 31);
            Piece x{row0 + us, u < to && !((shared_tiles >> u) & 1u) ? (int64_t)ut * BN_TILE + (lane & 7u) * 16 : K, {0, 0, 0, 0}};
            const uint8_t *const raw = a.raw + (a.ids ? srow : x.row) * K + x.col;
            if (wide && x.col < K) {
              const uint4 v = __ldg(reinterpret_cast<const uint4 *>(raw));
              x.rw[0] = v.x, x.rw[1] = v.y, x.rw[2] = v.z, x.rw[3] = v.w;
            } else if (x.col < K) {
#pragma unroll
              for (int i = 0; i < 4; i++)
                if (x.col + 4 * i < K) x.rw[i] = ldg_stream_u32(raw + 4 * i);
            }
            return x;
          };
          Piece next = fetch(from);
          for (int u0 = from; u0 < to; u0 += 4) {
            const Piece x = next;
            if (u0 + 4 < to) next = fetch(u0 + 4);
            if (x.col >= K) continue;
            const uint2 c = *reinterpret_cast<const uint2 *>(sc + (u0 + (int)(lane >> 3)) * TI_TILE + (lane & 7u) * 2);
            uint32_t o[8];
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const uint32_t cw = (i & 2 ? c.y : c.x) >> (16 * (i & 1));
              o[2 * i] = (__byte_perm(x.rw[i], 0u, 0x1100) & 0x807F807Fu) | pair[cw & 0xFFu];
              o[2 * i + 1] = (__byte_perm(x.rw[i], 0u, 0x3322) & 0x807F807Fu) | pair[(cw >> 8) & 0xFFu];
            }
            uint16_t *const dst = a.out + x.row * K + x.col;
            if (wide) {
              reinterpret_cast<uint4 *>(dst)[0] = make_uint4(o[0], o[1], o[2], o[3]);
              reinterpret_cast<uint4 *>(dst)[1] = make_uint4(o[4], o[5], o[6], o[7]);
            } else {
#pragma unroll
              for (int i = 0; i < 4; i++)
                if (x.col + 4 * i < K) *reinterpret_cast<uint2 *>(dst + 4 * i) = make_uint2(o[2 * i], o[2 * i + 1]);
            }
          }
          __syncwarp();  // the escaped weights' words are written over what went out above
          if (own && count) each_escape([&](uint32_t i, uint32_t e, uint32_t) {
            const int64_t col = (int64_t)t * BN_TILE + i;
            const uint32_t b = a.raw[srow * K + col];
            a.out[row * K + col] = (uint16_t)(((b & 0x80u) << 8) | (e << 7) | (b & 0x7Fu));
          });
          each_shared([&](int u, uint32_t nv, uint32_t ranks) {
            const int64_t col = (int64_t)__shfl_sync(BN_FULL, t, u) * BN_TILE + 4 * lane, r = row0 + __shfl_sync(BN_FULL, sub, u);
            if (!nv) return;
            const uint32_t b = ldg_stream_u32(a.raw + (a.ids ? srow : r) * K + col);
            const uint32_t e0 = tbl[ranks & 0xFFu], e1 = tbl[(ranks >> 8) & 0xFFu], e2 = tbl[(ranks >> 16) & 0xFFu], e3 = tbl[ranks >> 24];
            *reinterpret_cast<uint2 *>(a.out + r * K + col) = make_uint2((__byte_perm(b, 0u, 0x1100) & 0x807F807Fu) | (e0 << 7) | (e1 << 23), (__byte_perm(b, 0u, 0x3322) & 0x807F807Fu) | (e2 << 7) | (e3 << 23));
          });
        }
        from = to;
      }
      if (rows > 1 || rows_per_task > 1) break;
    }
    if (MODE == RICE_R4) {
      const bool leader = rows_per_task > 1 ? (int)lane < rows * T && (int)lane % T == 0 : lane == 0;
      if (leader) {
        const int64_t row = row0 + (rows_per_task > 1 ? (int)lane / T : 0);
        a.row_cnt[row] = row_escapes;
        escapes += row_escapes;
      }
    }
  }
  if (MODE == RICE_R4) {
    escapes = __reduce_add_sync(BN_FULL, escapes);
    if (lane == 0 && escapes) atomicAdd(a.counters + 2, escapes);
  }
}

template <int MODE>
int launch_tiles(const RiceArgs &a, uint8_t *slots, int64_t row_bytes, cudaStream_t s) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // rows spread evenly over sixteen blocks an SM, at most eight a block
  const int64_t spread = (a.R + (int64_t)sms * 16 - 1) / ((int64_t)sms * 16);
  const int per_block = (int)min((int64_t)8, max((int64_t)1, spread));
  rice_scan_kernel<MODE><<<(unsigned)((a.R + per_block - 1) / per_block), 32, (size_t)per_block * SC_STRIDE * 4, s>>>(a, slots, row_bytes, per_block);
  if (int e = launched("rice_scan_kernel")) return e;
  auto kern = rice_tiles_kernel<MODE>;
  BN_CUDA(allow_smem(kern, TI_SMEM));
  // as many rows a task as keep every warp at one task, up to the task's 32 tiles (one task of 32 tiles
  // takes about as long as one of three: 1000 x 128 16.4 -> 12.6 us, 20000 x 512 35 -> 35)
  const int64_t all_warps = (int64_t)sms * TI_WARPS;
  const int rows_per_task = a.ids || a.T > 16 ? 1 : (int)max((int64_t)1, min((int64_t)(32 / a.T), (a.R + all_warps - 1) / all_warps));
  const int64_t tasks = (a.R + rows_per_task - 1) / rows_per_task;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)min(tasks, (int64_t)sms)), cfg.blockDim = dim3(TI_WARPS * 32), cfg.dynamicSmemBytes = TI_SMEM, cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;  // the deposit table is built while the scan runs
  cfg.attrs = attr, cfg.numAttrs = 1;
  BN_CUDA(cudaLaunchKernelEx(&cfg, kern, a, (const uint8_t *)slots, row_bytes, rows_per_task));
  return launched("rice_tiles_kernel");
}

// Streams may start on any word (a shard uploaded whole, with pointers into it): `bits` is rounded
// down to the 16 bytes that the kernels read at a time, which stay inside the caller's allocation.
// false: outside the kernels' coverage.
bool tiles_cover(RiceArgs &a) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(a.bits);
  a.shift = (uint32_t)(at & 15) / 4;
  if (a.K % 4 || at & 3 || a.T > (1 << 18) || a.R > (1ll << 31) || (a.shift && a.nwords > 0xFFFFFFF0u)) return false;
  a.bits -= a.shift, a.nwords += a.shift;
  return true;
}

}  // namespace

int rice_tiles_r4(RiceArgs a, cudaStream_t s) {
  if ((reinterpret_cast<uintptr_t>(a.codes) & 7) || !tiles_cover(a)) return -1;
  return launch_tiles<RICE_R4>(a, reinterpret_cast<uint8_t *>(a.codes), (int64_t)a.T * 64, s);
}

int rice_tiles_unpack(RiceArgs a, cudaStream_t s) {
  if (((reinterpret_cast<uintptr_t>(a.raw) | reinterpret_cast<uintptr_t>(a.out)) & 15) || !tiles_cover(a)) return -1;
  return launch_tiles<RICE_UNPACK>(a, reinterpret_cast<uint8_t *>(a.out), a.K * 2, s);
}

}  // namespace bn
