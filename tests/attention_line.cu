// Host build of the rule that takes a call of the prompt attention op to one of its kernels, for test_attention_line.py.
#include "../megabake_b200/csrc/prompt_plan.h"

extern "C" int on_tcgen05(int head_dim, int queries, int keys, long long heads, int masked, int sms, int limited) {
  return mk::attention_on_tcgen05(head_dim, queries, keys, heads, masked != 0, sms, limited != 0);
}

extern "C" int mask_in_eights(int head_dim, int queries, int keys) { return mk::attention_mask_in_eights(head_dim, queries, keys); }
extern "C" int mask_in_tiles(int head_dim, int queries, int keys) { return mk::attention_mask_in_tiles(head_dim, queries, keys); }
