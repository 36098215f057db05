// The rules by which a call is sent to one form of a kernel or another where the choice changes its time only, never
// its result. Plain functions of sizes, so that they can be checked without a GPU. Times: B200, fp16 unless stated.
#pragma once

namespace b200ait {

// Attention, heads above 64 channels: one CTA per SM with four K / V stages instead of two CTAs with two each. Taken
// where a second CTA would find nothing to do. One query row against 4096 keys of 96 channels, two CTAs' form -> lone:
// 16 heads 49 -> 46 us, 64 heads 55 -> 48, 148 heads 57 -> 49; with 160 heads two CTAs on some SMs are ahead (92 -> 68).
inline bool attn_lone(long long items, int sms) { return items <= sms; }

}  // namespace b200ait
