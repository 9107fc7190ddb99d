// Batched solver of general river subgames (batch_solver.cu): many independent river
// subgames, each with its own 5-card board, pot, stack and bet tree (batch_tree.h), solved
// with per-hand regrets by one persistent kernel fed from a device work queue.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "batch_tree.h"

namespace prb {

constexpr int kBLive = 1081;   // hands that share no card with a 5-card board
constexpr int kBRow = 1088;    // per-hand rows, padded to a multiple of 32
constexpr int kBLists = 47;    // off-board cards
constexpr int kBListLen = 46;  // live hands holding one off-board card
constexpr int kBChunks64 = kBRow / 64;  // 64-hand chunks of the rank-order scan

// One subgame as the kernels see it.
struct BSub {
    unsigned long long board;
    int node_off, num_nodes;
    int edge_off;  // first regret row: rows of kBRow values, one per edge
    int num_edges, num_leaves;
    float pot;
};

constexpr int kBMaxGroups = 136;  // tie groups of the live hands: the most any 5-card board has,
constexpr int kBMaxRows = 917;    // and over its 47 card lists (both counted over all boards)

// Per-subgame hand layout, built on the device from the board. Hands are held in rank
// order ("positions"), weakest first, positions kBLive.. kBRow-1 are padding. The tie groups of each
// card list are numbered through ("rows"), lists in card order.
struct BPack {
    uint32_t rows[kBRow];            // row of the hand's group in its low card's list | in its high card's << 16
    uint32_t grp[kBRow];             // tie group | list of the low card << 16 | list of the high card << 24
    uint16_t hand[kBRow];            // colex hand index of each position (0xFFFF: padding)
    uint16_t clpos[kBLists][48];     // positions holding each off-board card, in rank order
    uint2 ends[kBLists + 1];         // per list, bit j: its j-th hand is the last of its group
    uint16_t lrow[48];               // first row of each list
    uint16_t pgrp[kBRow];            // tie group of each position | 0x8000 at the group's last position
    uint16_t last[kBMaxGroups + 4];  // last position of each tie group
    uint16_t num_groups, pad[3];
    uint16_t pos_of[1328];           // position of each colex hand (0xFFFF: blocked)
};

static_assert(offsetof(BPack, clpos) % 16 == 0 && sizeof(BPack) % 16 == 0 && sizeof(uint16_t[kBLists][48]) % 16 == 0 &&
                  sizeof(uint16_t[48]) % 8 == 0 && sizeof(uint16_t[kBMaxGroups + 4]) % 8 == 0 && kBListLen <= 64,
              "clpos to num_groups move as 8-byte words");

enum { kBModeCFR = 0, kBModeBR = 1, kBModeEval = 2 };

struct BLaunch {
    const BSub *subs;
    const BNode *nodes;
    const BPack *packs;
    const float *ranges;  // [subgame][2][kBRow], position order
    float *regrets;       // [edge row][kBRow]
    float *avg;           // [edge row][kBRow] (average-strategy sums) or null
    const int *order;     // work queue: subgame ids in schedule order
    int *head;            // queue head, zero before the launch
    int count;            // subgames in the queue
    int player;           // updating / best-responding player
    int use_average;      // BR / Eval: strategies from the average sums instead of regrets
    void *root_out;       // [subgame][kBRow] root values of `player` (V), or null
    void *sum_out;        // [subgame] sum over hands of range x root value (V), or null
    void *child_out;      // [subgame][8][kBRow] values of the root's children (V), or null
    const double *ranges64;  // double passes: [subgame][2][kBRow] opponent weights, or null (use ranges)
    int own_reach;        // CFR: average sums weighted by the updater's range (subgames inside a larger
                          // game, whose ranges change between iterations), not by 1
    const float *avg_weight;  // CFR: device scalar multiplying this pass's average-sum terms, or null (1)
};

// Builds the packs and position-order ranges of `count` subgames: ranges_in holds
// [subgame][2][1326] colex-order ranges.
cudaError_t launch_batch_setup(const BSub *subs, int count, BPack *packs, const float *ranges_in,
                               float *ranges_pos, int *err, cudaStream_t stream);

// One pass over the queue. K = hands per thread (2, 3 or 4); fp64 selects double
// arithmetic (best response and evaluation only). ctas = grid size (persistent CTAs).
// dense (K = 4 CFR passes in single precision only): the configuration with registers capped
// for 3 CTAs per SM; it expects groups of batch_dense_group() leaves.
cudaError_t launch_batch_pass(int mode, int K, int fp64, int avg, const BLaunch &a, int ctas, int max_leaves,
                              cudaStream_t stream, int dense = 0);

// A CFR pass over a queue of subgames whose tree is check, check, showdown (nodes: player 0's decision,
// player 1's, the showdown), without child or summed outputs. The queue head is not used.
cudaError_t launch_check_pass(int avg, const BLaunch &a, int sms, cudaStream_t stream);

// Adds 1 to the device scalar *w (the next iteration's average weight), on `stream`.
cudaError_t launch_weight_step(float *w, cudaStream_t stream);

// Threads per CTA and shared memory of a configuration.
int batch_threads(int K);
size_t batch_smem_bytes(int K, int fp64, int group_leaves);
int batch_group_leaves(int fp64);
// Leaf group of the dense K = 4 configuration (3 CTAs per SM fit in shared memory).
int batch_dense_group();
// Resident CTAs per SM the configuration allows (0 if it cannot launch).
int batch_ctas_per_sm(int mode, int K, int fp64, int avg);
// The same for the dense K = 4 CFR configuration.
int batch_dense_ctas_per_sm(int avg);

}  // namespace prb
