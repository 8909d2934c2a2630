// Slot counts of the SSSP scratch when a growth fails (csrc/sssp_scratch.h),
// over a buffer that stands in for device memory.
#include <cstdio>

#include "sssp_scratch.h"

namespace {

size_t room;  // largest buffer that can be had

struct FakeBuf {
  size_t bytes = 0;
  int ensure(size_t need) {  // frees before it allocates, as the engine's
    if (need <= bytes) return 0;
    bytes = 0;
    if (need > room) return -4;
    bytes = need;
    return 0;
  }
};

int failures = 0;
void check(bool ok, const char *what) {
  if (!ok) failures++, std::printf("FAILED: %s\n", what);
}

}  // namespace

int main() {
  for (size_t bits : {size_t(0), size_t(10)}) {
    fapk::SsspScratch<FakeBuf> s;
    auto covered = [&](size_t slot) {
      return s.tables.bytes >= s.slots * slot && s.bits.bytes >= s.slots * bits;
    };
    room = 1000;
    check(s.ensure(5, false, 100, bits) == 0 && s.slots == 5 && covered(100), "first slots");
    check(s.ensure(3, false, 100, bits) == 0 && s.slots == 5, "fewer slots keep the count");
    // another user of the tables asks for more than there is
    check(s.tables.ensure(2000) != 0 && s.tables.bytes == 0, "the growth fails");
    check(s.ensure(4, false, 100, bits) == 0 && s.slots >= 4 && covered(100), "slots after a failed growth");
    check(s.ensure(11, false, 100, bits) != 0 && covered(100), "no slots are counted when the own growth fails");
    check(s.ensure(2, false, 100, bits) == 0 && s.slots == 2 && covered(100), "slots after an own failed growth");
    // the bitmaps fail behind the tables
    if (bits > 0) {
      room = 1000;
      s = {};
      check(s.ensure(1, false, 100, bits) == 0, "one slot");
      check(s.ensure(9, false, 100, 200) != 0 && s.slots == 0, "the bitmaps fail");
      check(s.ensure(9, false, 100, bits) == 0 && s.slots == 9 && covered(100), "slots after failed bitmaps");
    }
    // the wide layout counts its own slots, and back
    s = {};
    check(s.ensure(4, false, 100, bits) == 0 && s.ensure(1, true, 200, bits) == 0 && covered(200), "wide slots");
    check(s.ensure(4, false, 100, bits) == 0 && s.slots >= 4 && covered(100), "narrow slots again");
  }
  if (failures == 0) std::printf("OK\n");
  return failures != 0;
}
