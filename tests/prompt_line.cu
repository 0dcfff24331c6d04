// Host build of the prompts' rule between CTAs on their own and pairs, for test_prompt_line.py.
#include "../megabake_b200/csrc/prompt_plan.h"

// Whether a CTA brings half of a tile's weight rows.
extern "C" int on_pairs(int tokens, int sms) {
  mk::PromptPhase p{};
  p.rows = 64;
  return mk::prompt_box_rows(p, mk::prompt_class(tokens, sms)) != p.rows;
}
