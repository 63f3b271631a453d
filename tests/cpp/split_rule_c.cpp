// C entry to the split-K rule (split_rule.h) for tests/test_split_rule.py.
#include "split_rule.h"

extern "C" int split_pays(int M, int N, int K, int sms) { return b200::mlp::split_pays(M, N, K, sms); }
