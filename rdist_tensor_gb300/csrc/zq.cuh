// Sample state of the breadth-first FP64 STS-CP draws (zq_sampler.cu), J_max
// entries each unless stated.
#pragma once
#include "common.cuh"

namespace exafac {

struct ZState {
    int64_t* xi = nullptr;      // J x (R rounded up to 4): the descent's vector, fixed point (pack_x)
    int8_t* rest = nullptr;     // J x (R rounded up to 4): h less its fixed point, 256ths of a unit
    double2* lh = nullptr;      // (low, high) of the current descent
    double* rinv = nullptr;     // 1 / root mass (scaled units)
    float2* err = nullptr;      // error bounds of (low, high)
    float* e0 = nullptr;        // error bound of one mass over the root mass
    float* n1 = nullptr;        // sum of |x'|
    int32_t* ex = nullptr;      // exponent of the vector's largest entry
    int64_t* node = nullptr;    // current node
    int32_t* order[2] = {nullptr, nullptr};  // slot -> sample, ordered by node (ping-pong)
    int32_t* v = nullptr;       // eigen-tree leaf
    int32_t* pick = nullptr;    // row within the leaf, -1 while not placed
    int32_t* redo = nullptr;    // marked for the depth-first kernel
    int32_t* redo_list = nullptr;
    int32_t* redo_count = nullptr;  // 1
    int32_t* near_list = nullptr;   // leaf reached, its row within the FP32 stage's bound of another (later: FP64 weight)
    int32_t* near_count = nullptr;  // 1
    int32_t* lost = nullptr;        // 1: a wait of this draw ran out, its later kernels do nothing
    // of two consecutive levels (ping-pong), per tile of 128 slots:
    uint32_t* mask[2] = {nullptr, nullptr};   // 4 words: went left (or stayed)
    int32_t* tcount[2] = {nullptr, nullptr};  // flags set
    uint32_t* runs[2] = {nullptr, nullptr};   // 4 words: a run of equal node starts here (bit 0 of a tile clear)
    int64_t* pref64 = nullptr;  // per tile: prefix of tcount (more tiles than shared memory takes)
    int64_t* off[2] = {nullptr, nullptr};  // slot ranges of a level's nodes (ping-pong)
    int32_t* tree_exp = nullptr;           // 2 N + 1: exponent of each tree's root diagonal, and Phi's
    uint4* nodes = nullptr;     // a level's left children as product operands (z_node_cap of them)
};

void zq_carve(Arena& a, ZState& b, int R, int64_t J, int64_t widest, int trees);

}  // namespace exafac
