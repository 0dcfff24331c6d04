// Host build of the prompts' rule between CTAs on their own and narrow pairs, for test_prompt_line.py.
#include "../megabake_b200/csrc/prompt_plan.h"

extern "C" int on_pairs(int kind, int tokens, int sms) { return mk::prompt_pairs(kind, mk::prompt_class(tokens, sms)); }
