// Sizes of the GEMMs' shared-memory rings.  Plain C++ without CUDA, so that the rules can be checked on the host.
//
// A waiter tells the fills of a ring slot apart by one bit, the parity of the slot's barrier: asked for the fill of one round
// while the fill of the round BEFORE has not completed, the barrier says yes (that parity passed two fills ago) and the waiter
// reads what lies there.  So whoever waits for a slot has to know that the slot's previous fill has completed.  One waiter
// that takes every slot in turn knows it from its own last wait.  Groups of warps that take turns do not: what a group knows
// is that the fills of its OWN earlier turns have completed, and bulk copies in flight complete in any order.
#pragma once

namespace b200gptq {

// One CTA per 128 columns (gemm.cu): a k-tile per stage, `groups` groups take k-tiles in turn.  With a multiple of `groups`
// stages a stage always belongs to one group, which saw its previous fill itself.
constexpr int ring_in_whole_turns(int stages, int groups) { return stages / groups * groups; }

// Pairs of CTAs (gemm_pair.cu): a slot of the weight ring holds two k-tiles, four groups take k-tiles in turn, through tiles
// of `k_tiles` whose last slot may hold one.  From one k-tile of a group to its next the slots move on by up to:
constexpr int kPairGroups = 4;
constexpr int pair_slot_step(int k_tiles) { return k_tiles == 1 ? kPairGroups : (k_tiles % 2 ? 3 : 2); }
// Where that is always 2, an even number of slots gives every slot to the same two groups: each saw the previous fill itself.
// Otherwise the warp that fills the ring starts a fill only when the one `ahead` before it has completed: a group that has
// seen fill u complete then knows it of all fills up to u - ahead; its next wait is for u + step at most, and the previous
// fill of that slot is u + step - slots.
constexpr int kPairNoLimit = 1 << 30;
constexpr int pair_fill_ahead(int slots, int step) { return step == 2 && slots % 2 == 0 ? kPairNoLimit : slots - step; }

constexpr int kPairColumns = 128, kPairKTile = 64;         // columns per CTA, rows of K per stage
constexpr int kPairTmemCols = 512;                         // accumulators, then 32 columns of A per stage
constexpr int kPairSmem = 222 * 1024;
constexpr int kPairMaxStages = 14, kPairMaxSlots = 16;

constexpr int pair_zero_words(int bits) { return bits % 4 == 0 ? 4 * bits : (4 * bits + 3 + 3) & ~3; }
constexpr int pair_unit_bytes(int bits) { return 4 * bits * kPairColumns * 4; }      // packed weights of 128 rows
// a slot of the weight ring: packed rows | scales [group][column] | zero-point words of each group
constexpr int pair_slot_bytes(int bits, int groups) { return pair_unit_bytes(bits) + groups * (kPairColumns * 2 + 128); }

struct PairRings {
    int acc_sets;      // sets of accumulators
    int stages;        // of x (shared memory) and A (tensor memory)
    int slots;         // of packed weights and constants
    int ahead;         // fills of the weight ring in flight at most
};
inline PairRings pair_rings(int bits, int groups, int rows, int k_tiles) {      // rows of x per tile
    PairRings r;
    r.acc_sets = rows <= 128 ? 2 : 1;
    r.stages = (kPairTmemCols - r.acc_sets * rows) / 32;
    if (r.stages > kPairMaxStages) r.stages = kPairMaxStages;
    r.slots = (kPairSmem - 1024 - r.stages * (rows / 2 * kPairKTile * 2)) / pair_slot_bytes(bits, groups);
    if (r.slots > kPairMaxSlots) r.slots = kPairMaxSlots;
    const int step = pair_slot_step(k_tiles);
    if (step == 2) r.slots &= ~1;
    r.ahead = pair_fill_ahead(r.slots, step);
    return r;
}

}  // namespace b200gptq
