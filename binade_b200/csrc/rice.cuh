// Arguments shared by the Rice stream decoders.
#pragma once

#include "common.cuh"

namespace bn {

enum RiceMode { RICE_RANKS = 0, RICE_UNPACK = 1, RICE_R4 = 2 };

struct RiceArgs {
  const uint8_t *meta;
  const uint32_t *bits;
  uint64_t nwords;
  uint32_t shift;  // the stream's first word is bits[shift]: `bits` rounded down to 16 bytes (rice_tiles.cu)
  const uint32_t *roff;
  const uint8_t *table;
  const uint8_t *raw;
  int64_t R, K;
  int T;
  // lookups (RICE_UNPACK only): output row i decodes stream row ids[i] of a table of `rows` rows
  const uint32_t *ids;
  int64_t rows;
  // format 1 (fixed-width codes, FMT == 1): `bits` is the index stream, `roff` the first word of
  // each row (bn_f1_offsets), f1_esc the file's escape bytes, f1_eoff the escapes before each row
  const uint8_t *f1_esc;
  uint64_t f1_nesc;
  const uint32_t *f1_eoff;
  // outputs
  uint32_t *ranks;   // RICE_RANKS: [R, T*32] four 8-bit ranks per word
  uint32_t *rend;    // RICE_RANKS / RICE_UNPACK: word after each row's last bit
  uint16_t *out;     // RICE_UNPACK: BF16 [R, K]
  uint16_t *codes;   // RICE_R4
  uint8_t *flags;    // RICE_R4
  uint32_t *row_cnt; // RICE_R4
  uint8_t *esc_tmp;  // RICE_R4 scratch
  uint64_t esc_cap;
  uint32_t *tmp_off;
  uint32_t *counters;
};

#ifdef __CUDACC__
// The low n bits: all of them from 32 on, none below 1.
__device__ __forceinline__ uint32_t low_mask(int n) {
  uint32_t m;
  asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(m) : "r"((uint32_t)max(n, 0)));
  return m;
}
#endif

// Decode in two kernels, one thread per tile (rice_tiles.cu); -1 when the arrays are outside their
// coverage. rice_tiles_r4 fills what rice_kernel<RICE_R4> fills, rice_tiles_unpack what
// rice_kernel<RICE_UNPACK> fills.
int rice_tiles_r4(RiceArgs a, cudaStream_t s);
int rice_tiles_unpack(RiceArgs a, cudaStream_t s);

}  // namespace bn
