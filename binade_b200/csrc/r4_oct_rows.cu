// Several input rows against R4 weights in the documented order: 2..8 rows of a linear layer, and the
// slots of an expert gather grouped by expert. The batch-1 kernel's decode (r4_oct.cu: eight threads
// per weight row, four rows a warp, private cp.async rings, escapes by column streams) with M
// accumulators per virtual lane: a tile is decoded once and multiplied by M input rows.
//
//   x        M rows as BF16 in shared memory, in the unused halves of the pair table's entries where
//            they fit (M T <= 128), else above the table; 32 bytes a thread, tile and row
//   grouped  blockIdx.y is the i-th group of up to M slots over all experts, found by a prefix sum of
//            the experts' group counts at block start; the grid holds the most groups there can be
//            (active experts + slots / M: 256 for the about 176 groups of 64 tokens, top 8 of 128),
//            and a block past the last group leaves at once; blocks of one group share an expert's
//            rows (grid.x)
//   half     a block with at most M / 2 input rows runs the code for M / 2
//   end of a row  the 4 M accumulators of a thread are summed over the row's eight threads while the
//            input rows are dealt out to them (16 shuffles instead of 48 for M = 4); additions pair
//            the same lanes as in the documented order, and a sum of two does not depend on which comes first
//
// Bound: instruction issue (per four rows and tile about 100 instructions of decode and 18 M of
// loads of x and products).
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "oct.cuh"

namespace bn {
namespace {

struct OctRowsArgs {
  bn_r4 w;
  const uint16_t *x;
  uint16_t *y, *y2;
  int64_t N, K;                // rows (of one expert, for a gather)
  int64_t x_stride, y_stride;  // elements between input rows / output rows
  int T, m;                    // input rows (plain)
  // grouped gather (seg != nullptr): an expert's slots are order[seg[e] .. seg[e + 1]), slot s
  // multiplies input row xi[s] by rows e * RS + R0 .. + N; outputs y [G, N], or with 0 < split < N
  // y [G, split] and y2 [G, N - split]
  const uint32_t *xi, *seg, *order;
  int64_t E, RS, R0, split;
  uint32_t smem;
};

__device__ int g_oct_rows_error;  // the shared window does not match the launch; read by bn_device_status()

constexpr int OR_ROUND = 4;  // rows a warp walks side by side
using Geo4 = OctGeom<4>;

// Bytes of a tile and of an input row in shared memory, and where the rows start.
template <bool HOLES>
struct XGeom {
  static constexpr uint32_t TILE = HOLES ? 512 : 256, HALF = HOLES ? 256 : 128;
};
__host__ __device__ inline uint32_t rows_x_bytes(bool holes, int M, int T) { return holes ? 0u : (uint32_t)M * (uint32_t)T * 256u; }

// One block's part of the work, for MM input rows (those past `count` are zeros).
template <int MM, int NQ, bool HOLES>
__device__ __forceinline__ void rows_body(const OctRowsArgs &a, uint32_t ring, uint32_t x_at, uint32_t lane, uint32_t gw, uint32_t nwarps, int64_t row0, int64_t g_first, int count, uint32_t ready, const uint8_t *praw0, const uint8_t *pcode0, uint32_t epos0, uint32_t col0, uint32_t flag0) {
  using X = XGeom<HOLES>;
  constexpr uint32_t SLOT = Geo4::SLOT, QUAD = Geo4::QUAD;
  const uint32_t p = lane & 7u, grp = lane >> 3;
  const int T = a.T;
  const int64_t K = a.K, N = a.N;
  const uint32_t G = (uint32_t)((N + OR_ROUND - 1) / OR_ROUND);
  const bool partial = (K & 127) != 0;
  const uint32_t pmax = (uint32_t)(K & 127) / 16u, row_codes = (uint32_t)T * 64u;
  const uint32_t to_codes = 512u - lane * 8u, lut = OC_LUT + lane * 4u;
  const uint32_t xrow = (uint32_t)T * X::TILE, xs0 = x_at + p * 16u;

  // load side (the caller has filled the ring with the first NQ quads of group gw)
  uint32_t pg = gw;
  int pt = NQ * 4;
  bool plive = true;
  const uint8_t *praw = praw0, *pcode = pcode0;
  uint32_t m_flag = flag0, m_epos = epos0, m_col = col0;
  auto aim = [&]() {
    const int64_t srow = row0 + min((int64_t)pg * OR_ROUND + grp, N - 1);
    praw = a.w.raw + srow * K + p * 16u;
    pcode = reinterpret_cast<const uint8_t *>(a.w.codes) + srow * row_codes + p * 8u;
    m_epos = __ldg(a.w.row_esc + srow);
    m_col = __ldg(reinterpret_cast<const uint32_t *>(a.w.col_esc + srow * 16) + p);
    m_flag = (int)p < T ? (uint32_t)__ldg(a.w.flags + srow * T + p) : 0u;
  };

  // decode side
  uint32_t cg = gw;
  int ct = 0;
  const uint8_t *c_flags = nullptr;
  uint32_t fm = 0, nflag = 0, xs = xs0;
  EscStream col[2];
  float acc[MM][4];
  auto begin_group = [&](uint32_t epos, uint32_t cols, uint32_t flag) {
    c_flags = a.w.flags + (row0 + min((int64_t)cg * OR_ROUND + grp, N - 1)) * T;
    nflag = flag, xs = xs0, ct = 0;
    stream_open(col[0], a.w.esc_cols, epos + (cols & 0xFFFFu));
    stream_open(col[1], a.w.esc_cols, epos + (cols >> 16));
#pragma unroll
    for (int m = 0; m < MM; m++)
#pragma unroll
      for (int i = 0; i < 4; i++) acc[m][i] = 0.0f;
  };
  begin_group(epos0, col0, flag0);

  auto end_group = [&]() -> bool {
    float v[MM][4];
#pragma unroll
    for (int m = 0; m < MM; m++)
#pragma unroll
      for (int i = 0; i < 4; i++) v[m][i] = acc[m][i];
    uint32_t first = 0;  // the input row whose sum ends up in this thread
#pragma unroll
    for (int o = 4, held = MM; o >= 1; o >>= 1, held = held > 1 ? held / 2 : 1) {
      if (held > 1) {
        const bool up = p & (uint32_t)o;
#pragma unroll
        for (int j = 0; j < held / 2; j++)
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float send = up ? v[j][i] : v[j + held / 2][i], keep = up ? v[j + held / 2][i] : v[j][i];
            v[j][i] = keep + __shfl_xor_sync(BN_FULL, send, o);
          }
        first += up ? held / 2 : 0;
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) v[0][i] = v[0][i] + __shfl_xor_sync(BN_FULL, v[0][i], o);
      }
    }
    const float sum = (v[0][0] + v[0][2]) + (v[0][1] + v[0][3]);
    const int64_t r = (int64_t)cg * OR_ROUND + grp;
    if ((p & (8u / MM - 1u)) == 0 && r < N && (int)first < count) {
      const uint16_t out = f32_to_bf16_bits(sum);
      if (a.seg) {
        const int64_t o = a.order[g_first + first];  // the slot this input row belongs to
        if (a.split > 0 && r >= a.split) a.y2[o * (N - a.split) + (r - a.split)] = out;
        else a.y[o * (a.split > 0 ? a.split : N) + r] = out;
      } else {
        a.y[(int64_t)first * a.y_stride + r] = out;
      }
    }
    cg += nwarps;
    if (cg >= G) return false;
    begin_group(m_epos, m_col, m_flag);  // fetched when the load side crossed into this group
    return true;
  };

  // the tile in slot U of the quad at `at`
  auto tile = [&](auto u_, uint32_t at, uint32_t xt, uint32_t token, bool flagged, bool live) {
    constexpr int U = decltype(u_)::value;
    uint32_t rr[4], cc[2], w[8];
    ring_read<4, U>(at, to_codes, token, rr, cc);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      w[2 * i] = (__byte_perm(rr[i], 0u, 0x1100) & 0x807F807Fu) | lut_read(__byte_perm(cc[i >> 1], lut, (i & 1) ? 0x7624 : 0x7604), ready);
      w[2 * i + 1] = (__byte_perm(rr[i], 0u, 0x3322) & 0x807F807Fu) | lut_read(__byte_perm(cc[i >> 1], lut, (i & 1) ? 0x7634 : 0x7614), ready);
    }
    if (flagged) {
      const uint32_t h0 = hits15(cc[0]), h1 = hits15(cc[1]);
      if (h0) stream_patch<0>(h0, col[0], a.w.esc_cols, w);
      if (h1) stream_patch<4>(h1, col[1], a.w.esc_cols, w);
    }
    if (!live) return;  // columns >= K are skipped, not added as zeros
#pragma unroll
    for (int m = 0; m < MM; m++) {
      uint32_t xx[8];
      asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4+%5];" : "=r"(xx[0]), "=r"(xx[1]), "=r"(xx[2]), "=r"(xx[3]) : "r"(xt + m * xrow), "n"(U * X::TILE), "r"(ready));
      asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4+%5];" : "=r"(xx[4]), "=r"(xx[5]), "=r"(xx[6]), "=r"(xx[7]) : "r"(xt + m * xrow), "n"(U * X::TILE + X::HALF), "r"(ready));
#pragma unroll
      for (int i = 0; i < 4; i++) acc[m][i] = fma2_bf16(w[2 * i + 1], xx[2 * i + 1], fma2_bf16(w[2 * i], xx[2 * i], acc[m][i]));
    }
  };
  using I0 = std::integral_constant<int, 0>;

  uint32_t at = ring;
  const uint32_t ring_end = ring + NQ * QUAD;
  for (;;) {
    if ((ct & 7) == 0) {  // a new block of eight tiles: fold the flag bytes, fetch the next block's
      const uint32_t v = __ballot_sync(BN_FULL, nflag != 0);
      fm = (v | (v >> 8) | (v >> 16) | (v >> 24)) & 0xFFu;
      const int nt = ct + 8 + (int)p;
      nflag = nt < T ? (uint32_t)__ldg(c_flags + nt) : 0u;
    }
    const uint32_t fq = fm >> (ct & 4);
    const int cn = min(4, T - ct), pn = plive ? min(4, T - pt) : 0;
    const uint32_t token = cp_wait<NQ - 1>();
    if (cn == 4 && !partial) {
      tile(I0(), at, xs, token, fq & 1u, true);
      tile(std::integral_constant<int, 1>(), at, xs, token, fq & 2u, true);
      tile(std::integral_constant<int, 2>(), at, xs, token, fq & 4u, true);
      tile(std::integral_constant<int, 3>(), at, xs, token, fq & 8u, true);
    } else {
      for (int u = 0; u < cn; u++) tile(I0(), at + u * SLOT, xs + u * X::TILE, token, (fq >> u) & 1u, !(partial && ct + u == T - 1) || p < pmax);
    }
    for (int u = 0; u < pn; u++) {
      const bool short_tile = partial && pt + u == T - 1 && p >= pmax;  // threads past the row's end copy thread 0's bytes and ignore them
      copy_tile<4, 0>(at + u * SLOT, to_codes, (short_tile ? praw - p * 16u : praw) + u * 128, pcode + u * 64, true, acc[0][0]);
    }
    cp_commit();
    praw += pn * 128, pcode += pn * 64, pt += pn;
    if (plive && pt == T) {
      pt = 0, pg += nwarps, plive = pg < G;
      if (plive) aim();
    }
    xs += cn * X::TILE, ct += cn;
    at = at + QUAD == ring_end ? ring : at + QUAD;
    if (ct == T && !end_group()) break;
  }
}

// M: most input rows a block multiplies by; NQ: quads of four tiles in a warp's ring; HOLES: x lives
// in the unused halves of the table's entries.
template <int M, int NQ, int MAXW, bool HOLES>
__global__ void __launch_bounds__(MAXW * 32, 1) r4_oct_rows_kernel(const __grid_constant__ OctRowsArgs a) {
  using X = XGeom<HOLES>;
  constexpr uint32_t QUAD = Geo4::QUAD;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ uint32_t s_tab[16];
  __shared__ int s_item[3];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, p = lane & 7u, grp = lane >> 3;
  const uint32_t W = blockDim.x >> 5, base = smem_addr(smem_raw);
  const int T = a.T;
  const int64_t K = a.K, N = a.N;
  OctLayout L = oct_layout(base, W, NQ * QUAD);
  const uint32_t x_bytes = rows_x_bytes(HOLES, M, T);
  if (base > OC_BASE_MAX || L.end + x_bytes > base + a.smem) {  // the host sized the window for another layout
    if (threadIdx.x == 0) atomicExch(&g_oct_rows_error, 1);
    return;
  }
  const uint32_t ring = (warp < L.in_a ? L.ring_a + warp * (NQ * QUAD) : OC_TOP + x_bytes + (warp - L.in_a) * (NQ * QUAD)) + lane * 16u;
  const uint32_t x_at = HOLES ? OC_LUT + 128u : OC_TOP;

  // this block's input rows and the storage row of its output row 0
  int64_t row0 = 0, g_first = 0;
  int count = a.m;
  if (a.seg) {
    pdl_wait();  // the slots' order is a kernel's output
    if (warp == 0) {
      int before = 0, item = (int)blockIdx.y, e_found = -1, chunk = 0;
      for (int64_t e0 = 0; e0 < a.E && e_found < 0; e0 += 32) {
        const int64_t e = e0 + lane;
        const int groups = e < a.E ? (int)((a.seg[e + 1] - a.seg[e] + M - 1) / M) : 0;
        int upto = groups;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int n = __shfl_up_sync(BN_FULL, upto, d);
          if (lane >= (uint32_t)d) upto += n;
        }
        const uint32_t holds = __ballot_sync(BN_FULL, before + upto > item);
        if (holds) {
          const int src = __ffs((int)holds) - 1;
          e_found = (int)e0 + src;
          chunk = item - (before + __shfl_sync(BN_FULL, upto - groups, src));
        } else {
          before += __shfl_sync(BN_FULL, upto, 31);
        }
      }
      if (lane == 0) s_item[0] = e_found, s_item[1] = chunk;
    }
    __syncthreads();
    const int e = s_item[0];
    if (e < 0) return;  // more blocks than groups
    g_first = (int64_t)a.seg[e] + (int64_t)s_item[1] * M;
    count = (int)min((int64_t)M, (int64_t)a.seg[e + 1] - g_first);
    row0 = (int64_t)e * a.RS + a.R0;
  }

  // the first NQ quads of this warp's first group, then x and the table
  const uint32_t G = (uint32_t)((N + OR_ROUND - 1) / OR_ROUND), nwarps = gridDim.x * W, gw = blockIdx.x * W + warp;
  const bool live = gw < G;
  const uint8_t *praw = nullptr, *pcode = nullptr;
  uint32_t epos = 0, cols = 0, flag = 0;
  if (live) {
    const int64_t srow = row0 + min((int64_t)gw * OR_ROUND + grp, N - 1);
    praw = a.w.raw + srow * K + p * 16u;
    pcode = reinterpret_cast<const uint8_t *>(a.w.codes) + srow * ((int64_t)T * 64) + p * 8u;
    epos = __ldg(a.w.row_esc + srow);
    cols = __ldg(reinterpret_cast<const uint32_t *>(a.w.col_esc + srow * 16) + p);
    flag = (int)p < T ? (uint32_t)__ldg(a.w.flags + srow * T + p) : 0u;
#pragma unroll
    for (int q = 0; q < NQ; q++) {  // (rows are longer than the ring: these are whole tiles)
#pragma unroll
      for (int u = 0; u < 4; u++) copy_tile<4, 0>(ring + q * QUAD + u * Geo4::SLOT, 512u - lane * 8u, praw + u * 128, pcode + u * 64, true, 0.0f);
      cp_commit();
      praw += 512, pcode += 256;
    }
  }
  pdl_launch_dependents();
  if (!a.seg) pdl_wait();  // x may be the previous kernel's output; the weights above are not
  {
    const uint32_t tab = threadIdx.x < 15 ? (uint32_t)__ldg(a.w.table + threadIdx.x) : 0u;
    const int rows = count <= M / 2 ? M / 2 : M, pieces = T * 16;  // 16-byte pieces of an input row
    for (int m = 0; m < rows; m++) {
      const int64_t xr = m >= count ? -1 : a.seg ? (int64_t)a.xi[a.order[g_first + m]] * K : (int64_t)m * a.x_stride;
      const uint4 *const src = reinterpret_cast<const uint4 *>(a.x + xr);
      for (int i = threadIdx.x; i < pieces; i += blockDim.x) {
        const uint4 v = xr >= 0 && (int64_t)i * 8 < K ? __ldg(src + i) : make_uint4(0, 0, 0, 0);
        // thread p of a row's eight reads values 16p .. 16p+7 at byte 16p of a tile's first half and
        // 16p+8 .. 16p+15 at byte 16p of its second
        const uint32_t t = (uint32_t)i >> 4, q = (uint32_t)i & 15u;
        *reinterpret_cast<uint4 *>(smem_raw + (x_at - base) + (uint32_t)m * (uint32_t)T * X::TILE + t * X::TILE + (q & 1u) * X::HALF + (q >> 1) * 16u) = v;
      }
    }
    if (threadIdx.x < 16) s_tab[threadIdx.x] = tab;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < 256 * 8; i += blockDim.x) {
      const uint32_t code = i >> 3, v = (s_tab[code & 15] << 7) | (s_tab[code >> 4] << 23);
      *reinterpret_cast<uint4 *>(smem_raw + (OC_LUT - base) + code * 256u + (i & 7u) * 16u) = make_uint4(v, v, v, v);
    }
    __syncthreads();
  }
  if (live) {
    uint32_t ready;
    asm volatile("mov.u32 %0, 0;" : "=r"(ready)::"memory");  // after the barrier: orders x / table reads
    if (count <= M / 2) rows_body<M / 2, NQ, HOLES>(a, ring, x_at, lane, gw, nwarps, row0, g_first, count, ready, praw, pcode, epos, cols, flag);
    else rows_body<M, NQ, HOLES>(a, ring, x_at, lane, gw, nwarps, row0, g_first, count, ready, praw, pcode, epos, cols, flag);
  }
  cp_wait<0>();
}

int rows_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// -1 when the window does not hold `warps` rings of NQ quads beside M rows of x.
template <int M, int NQ, int MAXW, bool HOLES>
int launch_rows_as(OctRowsArgs a, unsigned slices, unsigned items, unsigned warps, cudaStream_t s) {
  if (warps > MAXW || NQ * 4 >= a.T) return -1;  // the ring must be shorter than a row
  const uint32_t ring = NQ * Geo4::QUAD, x = rows_x_bytes(HOLES, M, a.T);
  const uint32_t e0 = oct_layout(0, warps, ring).end, e1 = oct_layout(OC_BASE_MAX, warps, ring).end;
  a.smem = (e0 > e1 ? e0 : e1) + x;
  if (a.smem > OC_SMEM_MAX) return -1;
  auto kern = r4_oct_rows_kernel<M, NQ, MAXW, HOLES>;
  BN_CUDA(allow_smem(kern, OC_SMEM_MAX));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(slices, items), cfg.blockDim = dim3(warps * 32), cfg.dynamicSmemBytes = a.smem, cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = 1;
  BN_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
  return launched("r4_oct_rows_kernel");
}

// As many warps as the registers of M accumulators and the shared window allow, spread evenly over
// the rows of a slice.
template <int M, int MAXW>
int launch_rows(const OctRowsArgs &a, int64_t slices, int64_t items, cudaStream_t s) {
  const int64_t groups = (a.N + OR_ROUND - 1) / OR_ROUND;
  if (slices > groups) slices = groups;
  for (int most = MAXW; most >= 8; most -= 2) {
    const int64_t rounds = (groups + slices * most - 1) / (slices * most), warps = (groups + slices * rounds - 1) / (slices * rounds);
    int e = -1;
    if (M * a.T <= 128) {  // 256 halves of table entries, two a tile
      e = launch_rows_as<M, 2, MAXW, true>(a, (unsigned)slices, (unsigned)items, (unsigned)warps, s);
      if (e == -1) e = launch_rows_as<M, 1, MAXW, true>(a, (unsigned)slices, (unsigned)items, (unsigned)warps, s);
    } else {
      e = launch_rows_as<M, 2, MAXW, false>(a, (unsigned)slices, (unsigned)items, (unsigned)warps, s);
      if (e == -1) e = launch_rows_as<M, 1, MAXW, false>(a, (unsigned)slices, (unsigned)items, (unsigned)warps, s);
    }
    if (e != -1) return e;
  }
  return -1;
}

bool rows_cover(const bn_r4 *w, const uint16_t *x, int64_t N, int64_t K) {
  if (K % 16 || K < 640 || K > 16384 || N < 1 || N > (1ll << 30) || !w->esc_cols || !w->col_esc) return false;
  return ((reinterpret_cast<uintptr_t>(w->raw) | reinterpret_cast<uintptr_t>(w->codes) | reinterpret_cast<uintptr_t>(x)) & 15) == 0 && ((reinterpret_cast<uintptr_t>(w->esc_cols) | reinterpret_cast<uintptr_t>(w->col_esc)) & 3) == 0;
}

}  // namespace

int oct_rows_status(int *status) {
  BN_CUDA(cudaMemcpyFromSymbol(status, g_oct_rows_error, sizeof(int)));
  return BN_OK;
}
int oct_rows_status_reset() {
  const int zero = 0;
  BN_CUDA(cudaMemcpyToSymbol(g_oct_rows_error, &zero, sizeof(int)));
  return BN_OK;
}

int oct_rows(const bn_r4 *w, const uint16_t *x, int64_t x_stride, int64_t M, int64_t N, int64_t K, uint16_t *y, int64_t y_stride, cudaStream_t s) {
  if (M < 2 || M > 8 || x_stride % 8 || !rows_cover(w, x, N, K)) return -1;
  OctRowsArgs a{};
  a.w = *w, a.x = x, a.y = y, a.N = N, a.K = K, a.T = (int)tiles(K), a.m = (int)M, a.x_stride = x_stride, a.y_stride = y_stride;
  const int64_t blocks = rows_sms();
  // four rows a warp need rows for seven warps an SM; below, the bulk-copy kernel is faster (us with
  // two input rows, that kernel / this: 2048 x 3840 9.9 / 11.1, 3840 x 15360 40.6 / 42.1, 4096 x
  // 3840 14.3 / 11.8, 15360 x 3840 36.1 / 23.4)
  if (N < blocks * 27) return -1;
  // a thread applies its columns' escapes one after the other, which the few warps of few weight rows do not
  // hide: from a share of the weights that grows with the rows an SM has, the bulk-copy kernel is faster
  // (us, this / that with two input rows: 4096 x 3840, a fifth escaped 31 / 35, 28 % 39 / 37; 8192 x 2048, half
  // 34 / 39, 70 % 44 / 39; 15360 x 3840, 94 % 149 / 172; with eight, half escaped 189 / 179)
  const double escaped = (double)w->n_esc / ((double)N * (double)K), rows_an_sm = (double)N / (double)blocks;
  if (escaped > rows_an_sm / 110 || (M > 4 && escaped > 0.5)) return -1;
  return M == 2 ? launch_rows<2, 26>(a, blocks, 1, s) : M <= 4 ? launch_rows<4, 26>(a, blocks, 1, s) : launch_rows<8, 16>(a, blocks, 1, s);
}

int oct_gather_grouped(const bn_r4 *w, const uint16_t *x, const uint32_t *xi, const uint32_t *seg, const uint32_t *order, int64_t E, int64_t G, int64_t n, int64_t K, int64_t RS, int64_t R0, int64_t split, uint16_t *y, uint16_t *y2, cudaStream_t s) {
  if (E < 1 || E > (1 << 20) || G < 1 || !rows_cover(w, x, n, K)) return -1;
  OctRowsArgs a{};
  a.w = *w, a.x = x, a.y = y, a.y2 = y2, a.N = n, a.K = K, a.T = (int)tiles(K);
  a.xi = xi, a.seg = seg, a.order = order, a.E = E, a.RS = RS, a.R0 = R0, a.split = split;
  const int64_t active = G < E ? G : E;  // experts with work: at most one per slot
  // groups of four up to six slots an expert on average, else of eight (us, gate and up of 128
  // experts of 2 x 704 x 2816: 4 slots an expert 396 / 441, 2 slots 284 / 350; of 32 experts of 2 x
  // 1024 x 2048 with 8 slots each 236 / 216)
  const int wanted = G <= 6 * active ? 4 : 8;
  // fewer where the input rows' x does not fit the window (K = 16384: two)
  for (int m = wanted; m >= 2; m /= 2) {
    const int64_t most = active + G / m;
    if (most > 65535) return -1;
    // rows of an expert in as many slices as make the waves of blocks come out shortest: a wave takes
    // the rows of a slice and a start (table, x), which weighs as much as 170 row groups' tiles
    const double items = active * 0.45 + (double)G / m, start = 170.0 / ((double)((n + 3) / 4) * a.T);
    int64_t slices = 1;
    double best = 1e30;
    for (int64_t c = 1; c <= 24; c++) {
      const double cost = ceil(items * c / rows_sms()) * (1.0 / c + start);
      if (cost < best) best = cost, slices = c;
    }
    const int e = m == 8 ? launch_rows<8, 16>(a, slices, most, s) : m == 4 ? launch_rows<4, 24>(a, slices, most, s) : launch_rows<2, 26>(a, slices, most, s);
    if (e != -1) return e;
  }
  return -1;
}

}  // namespace bn
