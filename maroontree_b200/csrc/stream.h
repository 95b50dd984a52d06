// The encoder's entropy coding on the device (stream.cu): from the blocks'
// decisions and levels to the bytes of every tile.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace mth {

// The frame: 8x8 blocks in raster order, uniform tiles of tile_w8 x tile_h8
// blocks (the last of a row or column smaller).
struct StreamGeom {
  int w8 = 0, h8 = 0;    // frame size in samples (multiples of 8)
  int nbx = 0, nby = 0;  // in 8x8 blocks
  int sub = 0;           // 2: 4:2:0, 0: 4:4:4
  int sb_cols = 0, sb_rows = 0;
  int tile_w8 = 0, tile_h8 = 0;
  int tcols = 0, trows = 0;
};

struct StreamInput {
  const uint8_t* mode;  // luma mode of each block
  const uint8_t* tx;    // luma transform type of each block
  const int32_t* lv[3];  // levels: 64 per block in luma, 16 (4:2:0) or 64 in chroma
};

// One tile's extent in the token and digit buffers and its payload.
struct StreamTile {
  uint32_t base;    // first token (a multiple of kGroupTokens)
  uint32_t ntok;    // tokens, cdef_idx places included
  uint32_t shift;   // bits the range coder shifts out over the tile
  uint32_t digit;   // first 16-bit digit
  uint32_t byte;    // first byte of the payload in the payload buffer
  uint32_t nbytes;  // payload bytes
};

struct StreamTotals {
  uint32_t tokens;  // padded token buffer length
  uint32_t digits;  // 16-bit digits of all tiles
  uint32_t bytes;   // payload bytes of all tiles
  uint32_t pad;
};

// Buffer sizes.  `plan`: per-block counts and offsets and the tile table;
// `tokens(n)`: everything that grows with the padded token count;
// `digits(t)`: the coder's output.
size_t stream_plan_bytes(const StreamGeom& g);
size_t stream_token_bytes(const StreamGeom& g, uint32_t padded_tokens);
size_t stream_digit_bytes(const StreamTotals& t);
// The frame-initial CDFs of the symbols the encoder codes: bytes and the host
// copy for a quantiser context and chroma format.
size_t stream_cdf_bytes();
const void* stream_cdf_table(int qctx, int sub);

// Step 1: every block's token count, its context bytes and the offsets; the
// totals land in plan memory (stream_totals / stream_tiles give the device
// addresses).
int stream_count(const StreamGeom& g, const StreamInput& in, void* plan, cudaStream_t st, int* launches);
const StreamTotals* stream_totals(const StreamGeom& g, void* plan);
const StreamTile* stream_tiles(const StreamGeom& g, void* plan);
// Step 2: the tokens, partitioned by CDF, and the CDF adaptation: every
// token's store of the range coder.
int stream_trace(const StreamGeom& g, const StreamInput& in, void* plan, void* tokens, uint32_t padded_tokens,
                 const void* d_cdfs, bool updating, cudaStream_t st, int* launches);
// Step 3: the cdef_idx literals (*bits wide, one per 64x64 unit of `grid`;
// bits null: none) put in their places, and the coder's state at every piece
// of the store sequence; fills shift / digit / byte / nbytes and the totals.
int stream_ranges(const StreamGeom& g, void* plan, void* tokens, uint32_t padded_tokens, const int32_t* bits,
                  const uint8_t* grid, cudaStream_t st, int* launches);
// Step 4: the payload bytes of all tiles; `digits` holds stream_digit_bytes
// bytes, the longest payload has max_bytes bytes, and the payloads start at
// the returned address.
const uint8_t* stream_bytes(const StreamGeom& g, void* plan, void* tokens, uint32_t padded_tokens, void* digits,
                            const StreamTotals& t, uint32_t max_bytes, cudaStream_t st, int* launches);

}  // namespace mth
