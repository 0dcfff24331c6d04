// Host build of the order in which a prompt projection's CTA waits for its pipeline slots before it leaves, for
// test_prompt_drain.py.
#include "../megabake_b200/csrc/prompt_plan.h"

// How many uses have been consumed, in order, when the walk lets the CTA leave.  It begins with the fewest that a producer knows
// of: it has waited for the slot of its own last use, which may be the last but one of all (`uses` counts both producers').
extern "C" int uses_consumed_when_left(int uses, int stages) {
  int consumed = uses - 1 - stages > 0 ? uses - 1 - stages : 0;
  mk::prompt_drain(uses, stages, [&](int slot, uint32_t parity) {
    // a barrier's wait passes while the phase before the current one has the parity asked for
    auto phases = [&] { return consumed / stages + (consumed % stages > slot ? 1 : 0); };
    while ((phases() & 1) == static_cast<int>(parity) && consumed < uses) ++consumed;
    return true;
  });
  return consumed;
}
