// Which pressure solves may be in flight together on one GPU.  Blocks of a solve wait for one
// another, so all of them have to become resident whatever the others' places are.
#pragma once
#include <algorithm>

namespace bnn {

// A share of an SM is counted in units of 1/840 (840 is divisible by every resident-block count
// 1..8).
constexpr long long kShareUnits = 840;

// The launches of solves in flight, or one launch.  A block of k_pcg_chunk takes an SM to itself (its
// shared memory); blocks of the other kernels share SMs.
struct CoopLoad {
    int whole = 0;         // SMs taken by blocks that need one to themselves
    int blocks = 0;        // blocks that share SMs
    long long shared = 0;  // their units
    CoopLoad operator+(const CoopLoad& o) const { return {whole + o.whole, blocks + o.blocks, shared + o.shared}; }
    CoopLoad operator-(const CoopLoad& o) const { return {whole - o.whole, blocks - o.blocks, shared - o.shared}; }
};

// Blocks of the sharing kind alone fill up the SMs wherever they lie.  Beside them a block that
// needs an empty SM may find one of theirs on every SM: there must be an SM for each block of
// either kind.
inline bool coop_fits(const CoopLoad& all, int numSM) {
    if(all.whole == 0) return all.shared <= numSM * kShareUnits;
    return all.whole + std::min(all.blocks, numSM) <= numSM;
}

} // namespace bnn
