// The attention kernel's plan of last rounds dealt out by key blocks, for test_split_plan.py.
#include "../sageattention_b200/csrc/sage3_split.h"

extern "C" {
// out: whole pairs, slots, blocks per slot, blocks of slot 0, rest0
void split_plan(int causal, int BHq, int nqt, int Nk, int shift, int D, int sms, int* out, uint32_t* first) {
    const sage3::SplitPlan p = causal ? sage3::plan_split<true>(BHq, nqt, Nk, shift, D, sms) : sage3::plan_split<false>(BHq, nqt, Nk, shift, D, sms);
    const int v[5] = {p.whole, p.slots, p.blocks, p.rest, p.rest0};
    for (int i = 0; i < 5; ++i) out[i] = v[i];
    for (int i = 0; i < p.slots; ++i) first[i] = p.first[i];
}
void split_tile(int causal, int j, int nqt, int BHq, int whole, int rest0, int* out) {
    if (causal) sage3::rest_tile<true>(j, nqt, BHq, whole, rest0, out[0], out[1]);
    else sage3::rest_tile<false>(j, nqt, BHq, whole, rest0, out[0], out[1]);
}
int split_walk(int causal, int BHq, int nqt, int sms) { return causal ? sage3::longest_walk<true>(BHq, nqt, sms) : sage3::longest_walk<false>(BHq, nqt, sms); }
int split_blocks(int causal, int mt, int Nk, int shift) {
    return causal ? sage3::tile_blocks<true>(mt, Nk, shift) : sage3::tile_blocks<false>(mt, Nk, shift);
}
}
