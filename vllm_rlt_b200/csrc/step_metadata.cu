// A step's metadata on the host: what the engine hands to the layers about every row and sequence, written straight into the pinned buffer
// that is uploaded.  Over Python lists the 16384 tokens of a step took 7 ms, as long as the layers they run through; over whole tensors still
// 0.3 ms of small operations, which a single user's step of 0.4 ms waited for.  This takes 30 us and 2 us.
#include <string.h>

#include <algorithm>

#include "common.cuh"

extern "C" RLT_API int rlt_step_metadata(int32_t* words, const int64_t* at, const int64_t* records, int portions, int sequences, int planes, int width,
                                         int short_sequences, int64_t rows, int64_t dummy_slot) {
  enum { kTokens, kPositions, kRowSeq, kPrevious, kCu, kLongCu, kStarts, kLengths, kSlots, kTables };
  RLT_REQUIRE(words != nullptr && at != nullptr && (portions == 0 || records != nullptr), "step_metadata: missing buffer");
  RLT_REQUIRE(portions >= 0 && portions <= sequences && planes >= 1 && width >= 0 && short_sequences >= 0 && short_sequences <= sequences,
              "step_metadata: bad counts");
  const int record = 5 + 2 * planes;
  RLT_REQUIRE(rows >= 0 && rows <= 0x7fffffff, "step_metadata: bad counts");
  for (int i = kTokens; i <= kTables; ++i) RLT_REQUIRE(at[i] >= 0, "step_metadata: an offset in front of the words");
  RLT_REQUIRE((reinterpret_cast<uintptr_t>(words + at[kTokens]) & 7u) == 0, "step_metadata: tokens need 8-byte alignment");
  int64_t needed = sequences - portions;
  for (int i = 0; i < portions; ++i) {
    const int64_t* r = records + static_cast<int64_t>(i) * record;
    RLT_REQUIRE(r[0] != 0 && r[1] >= 1, "step_metadata: a portion without tokens");
    RLT_REQUIRE(r[1] <= rows && r[2] >= 0 && r[2] <= 0x7fffffff - r[1], "step_metadata: positions beyond 32 bits");
    for (int plane = 0; plane < planes; ++plane)
      RLT_REQUIRE(r[6 + 2 * plane] >= 0 && (r[6 + 2 * plane] == 0 || r[5 + 2 * plane] != 0), "step_metadata: a page table without pages");
    needed += r[1];
  }
  RLT_REQUIRE(needed == rows, "step_metadata: the rows are not the portions' and the padding's");
  int64_t* tokens = reinterpret_cast<int64_t*>(words + at[kTokens]);
  int32_t *positions = words + at[kPositions], *row_seq = words + at[kRowSeq], *previous = words + at[kPrevious], *cu = words + at[kCu];
  int32_t row = 0;
  cu[0] = 0;
  for (int s = 0; s < sequences; ++s) {
    const int64_t* r = records + static_cast<int64_t>(s) * record;
    const bool padding = s >= portions;                    // a row of its own that belongs to nobody
    const int64_t* from = padding ? nullptr : reinterpret_cast<const int64_t*>(r[0]);
    const int32_t count = padding ? 1 : static_cast<int32_t>(r[1]), start = padding ? 0 : static_cast<int32_t>(r[2]);
    if (padding) tokens[row] = 0;
    else memcpy(tokens + row, from, static_cast<size_t>(count) * sizeof(int64_t));
    previous[row] = padding ? -1 : static_cast<int32_t>(r[4]);
    for (int32_t i = 0; i < count; ++i) {
      positions[row + i] = start + i;
      row_seq[row + i] = padding ? -1 : s;
    }
    for (int32_t i = 1; i < count; ++i) previous[row + i] = static_cast<int32_t>(from[i - 1]);
    row += count;
    cu[s + 1] = row;
    words[at[kStarts] + s] = start;
    words[at[kLengths] + s] = padding ? 0 : start + count;
    words[at[kSlots] + s] = static_cast<int32_t>(padding ? dummy_slot : r[3]);
    for (int plane = 0; plane < planes; ++plane) {
      int32_t* table = words + at[kTables] + (static_cast<int64_t>(plane) * sequences + s) * width;
      const int64_t pages = padding ? 0 : std::min<int64_t>(r[6 + 2 * plane], width);
      if (pages > 0) memcpy(table, reinterpret_cast<const int32_t*>(r[5 + 2 * plane]), static_cast<size_t>(pages) * sizeof(int32_t));
      std::fill(table + pages, table + width, 0);
    }
  }
  for (int s = short_sequences; s <= sequences; ++s) words[at[kLongCu] + s - short_sequences] = cu[s] - cu[short_sequences];
  return RLT_OK;
}
