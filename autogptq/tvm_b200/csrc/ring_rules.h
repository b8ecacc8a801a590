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

// Pairs of CTAs (gemm_pair.cu): units of two k-tiles, through one tile after the other; a tile with an odd number of k-tiles ends in
// a unit of one.  A slot of the weight ring holds a unit, and with a multiple of the groups a slot always belongs to one group, which
// saw its previous fill itself.  A stage (x and A) holds a unit as well; `stages` counts its k-tiles.  A group's turns are four units
// apart and products retire in order, so a wait for a stage knows that its products of two rounds before have retired if there are
// four units or more.
constexpr int kPairGroups = 4, kPairMinStages = 8;
constexpr int pair_turns(int k_tiles) { return (k_tiles + 1) & ~1; }

constexpr int kPairColumns = 128, kPairKTile = 64;         // columns per CTA, rows of K of a k-tile (a stage holds two)
constexpr int kPairTmemCols = 512;                         // accumulators, then 32 columns of A per k-tile of a stage
constexpr int kPairSmem = 222 * 1024;
constexpr int kPairMaxStages = 14, kPairMaxSlots = 16;

constexpr int pair_zero_words(int bits) { return bits % 4 == 0 ? 4 * bits : (4 * bits + 3 + 3) & ~3; }
constexpr int pair_unit_bytes(int bits) { return 4 * bits * kPairColumns * 4; }      // packed weights of 128 rows
// a slot of the weight ring: packed rows | scales [group][column] | zero-point words of each group
constexpr int pair_slot_bytes(int bits, int groups) { return pair_unit_bytes(bits) + groups * (kPairColumns * 2 + 128); }

struct PairRings {
    int acc_sets;      // sets of accumulators
    int stages;        // of x (shared memory) and A (tensor memory), in k-tiles: an even number
    int slots;         // of packed weights and constants
};
inline PairRings pair_rings(int bits, int groups, int rows, bool several_tiles = true) {      // rows of x per tile
    PairRings r;
    r.acc_sets = rows <= 128 && several_tiles ? 2 : 1;
    r.stages = (kPairTmemCols - r.acc_sets * rows) / 32;
    if (r.stages > kPairMaxStages) r.stages = kPairMaxStages;
    // A group of weight warps wants two slots, one to unpack and one to fill: a stage above the least gives way to that.
    for (r.stages &= ~1;; r.stages -= 2) {
        r.slots = (kPairSmem - 1024 - r.stages * (rows / 2 * kPairKTile * 2)) / pair_slot_bytes(bits, groups);
        if (r.slots > kPairMaxSlots) r.slots = kPairMaxSlots;
        r.slots = ring_in_whole_turns(r.slots, kPairGroups);
        if (r.slots >= 2 * kPairGroups || r.stages <= kPairMinStages) break;
    }
    return r;
}

}  // namespace b200gptq
