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
  int nbx = 0, nby = 0;  // in 8x8 blocks
  int sub = 0;           // 2: 4:2:0, 0: 4:4:4
  int sb_cols = 0, sb_rows = 0;
  int tile_w8 = 0, tile_h8 = 0;
  int tcols = 0, trows = 0;
  // What a group of tiles is kept to (18 GB of buffers); a tile alone may pass it.
  uint32_t max_tokens = 1u << 30;
};

struct StreamInput {
  const uint8_t* mode;  // luma mode of each block
  const uint8_t* tx;    // luma transform type of each block
  const int32_t* lv[3];  // levels: 64 per block in luma, 16 (4:2:0) or 64 in chroma
};

// One tile's extent in the token and digit buffers and its payload.
struct StreamTile {
  uint32_t base;    // first token in its group's buffer (a multiple of kGroupTokens; 0: a group starts)
  uint32_t ntok;    // tokens, cdef_idx places included
  uint32_t shift;   // bits the range coder shifts out over the tile
  uint32_t digit;   // first 16-bit digit in its group's buffer
  uint32_t byte;    // first byte of the payload in its group's payload buffer
  uint32_t nbytes;  // payload bytes
};

struct StreamTotals {
  uint32_t tokens;  // padded token buffer length of the largest group
  uint32_t digits;  // 16-bit digits of a group's tiles
  uint32_t bytes;   // payload bytes of a group's tiles
  uint32_t groups;
};

// Consecutive tiles that go through steps 2 to 4 together, in buffers of their
// size.  A frame is one group unless it has more tokens than max_tokens.
struct StreamGroup {
  int tile0 = 0, ntiles = 0;
  uint32_t tokens = 0;  // padded token buffer length
};
// The group that starts at tile0, from the host's copy of the tile table.
StreamGroup stream_group(const StreamTile* tiles, int ntiles, int tile0);

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

// Step 1: every block's token count, its context bytes and the offsets
// (stream_place, from the counts at stream_counts); the totals and the tiles'
// extents land in plan memory (stream_totals / stream_tiles give the device
// addresses).
int stream_count(const StreamGeom& g, const StreamInput& in, void* plan, cudaStream_t st, int* launches);
int stream_place(const StreamGeom& g, void* plan, cudaStream_t st, int* launches);
uint32_t* stream_counts(const StreamGeom& g, void* plan);
const StreamTotals* stream_totals(const StreamGeom& g, void* plan);
const StreamTile* stream_tiles(const StreamGeom& g, void* plan);
// Step 2: a group's tokens, partitioned by CDF, and the CDF adaptation: every
// token's store of the range coder.
int stream_trace(const StreamGeom& g, const StreamInput& in, void* plan, void* tokens, const StreamGroup& grp,
                 const void* d_cdfs, bool updating, cudaStream_t st, int* launches);
// Step 3: the cdef_idx literals (*bits wide, one per 64x64 unit of `grid`;
// bits null: none) put in their places, and the coder's state at every piece
// of the store sequence; fills the group's shift / digit / byte / nbytes and
// digit and byte totals.
int stream_ranges(const StreamGeom& g, void* plan, void* tokens, const StreamGroup& grp, const int32_t* bits,
                  const uint8_t* grid, cudaStream_t st, int* launches);
// Step 4: the payload bytes of the group's tiles; `digits` holds
// stream_digit_bytes bytes, the longest payload has max_bytes bytes, and the
// payloads start at the returned address.
const uint8_t* stream_bytes(const StreamGeom& g, void* plan, void* tokens, const StreamGroup& grp, void* digits,
                            const StreamTotals& t, uint32_t max_bytes, cudaStream_t st, int* launches);

}  // namespace mth
