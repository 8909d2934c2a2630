// sssp_scratch.h -- scratch of the batched SSSP, counted in slots (one per CTA).
//
// The table buffer is shared: the search with one CTA per source grows it too.
// A buffer that fails to grow has been freed, so the count kept here is only
// ever as good as the bytes that the buffers hold, and is checked against them
// on every call.
#pragma once

#include <algorithm>
#include <cstddef>

namespace fapk {

// Buf: bytes held, and ensure(bytes), which keeps or replaces the buffer and
// returns 0, or fails and leaves it empty.
template <typename Buf>
struct SsspScratch {
  Buf tables;         // slots x slot_bytes
  Buf bits;           // slots x bits_bytes: bitmaps that shared memory does not hold
  int slots = 0;      // slots of the layout last asked for
  bool wide = false;  // ... which is that of the FP64 search with 32 lanes

  // At least `want` slots of a layout.
  int ensure(int want, bool layout, size_t slot_bytes, size_t bits_bytes) {
    size_t held = tables.bytes / std::max<size_t>(slot_bytes, 1);
    if (bits_bytes > 0) held = std::min(held, bits.bytes / bits_bytes);
    slots = (int)(layout == wide ? std::min((size_t)slots, held) : held);
    wide = layout;
    if (want <= slots) return 0;
    slots = 0;
    int rc = tables.ensure(slot_bytes * want);
    if (rc == 0) rc = bits.ensure(std::max<size_t>(bits_bytes * want, 4));
    if (rc == 0) slots = want;
    return rc;
  }
};

}  // namespace fapk
