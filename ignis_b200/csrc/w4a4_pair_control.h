// What the W4A4 pair kernel (nvfp4_w4a4.cu) keeps in shared memory behind its ring: the barriers, then the word that
// tcgen05.alloc writes the tensor-memory base to. Plain C++, so that a host test can check it. The offsets come from one
// struct: placed by hand, the slot once lay on the last of the barriers that had been added in front of it.
#ifndef B200Q_W4A4_PAIR_CONTROL_H
#define B200Q_W4A4_PAIR_CONTROL_H

#include <cstddef>
#include <cstdint>

namespace b200q {

constexpr int kPairStages = 5;

struct PairControl {
  uint64_t full[kPairStages];       // the first CTA's: a stage's bytes of both CTAs have landed
  uint64_t empty[kPairStages];      // the MMAs that read a stage have retired
  uint64_t acc_full;                // a tile's MMAs have retired
  uint64_t acc_empty;               // the first CTA's: both CTAs have pulled the tile out of tensor memory
  uint64_t sf_ready[kPairStages];   // the first CTA's: a stage's scales are in both CTAs' tensor memory
  uint32_t tmem_slot;
};
constexpr uint32_t kPairControlBytes = 256;   // kept for it
static_assert(sizeof(PairControl) <= kPairControlBytes, "barriers and slot fit the bytes kept for them");

constexpr uint32_t kPairFull = offsetof(PairControl, full), kPairEmpty = offsetof(PairControl, empty), kPairAccFull = offsetof(PairControl, acc_full),
                   kPairAccEmpty = offsetof(PairControl, acc_empty), kPairSfReady = offsetof(PairControl, sf_ready),
                   kPairTmemSlot = offsetof(PairControl, tmem_slot);
static_assert(kPairTmemSlot >= kPairSfReady + 8u * kPairStages, "the slot lies behind every barrier");

}  // namespace b200q

#endif
