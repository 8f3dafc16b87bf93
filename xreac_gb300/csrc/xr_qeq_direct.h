// The QEq solver for systems whose whole matrix fits one block's shared memory (xr_qeq_direct.cu).
#pragma once

#include "xr_common.cuh"

// Nine tile rows of 32: 45 tiles of the lower triangle and 8 scratch tiles, 212 of the 227 KB a block may have.
constexpr int kQeqDirectMax = 288;
// Systems of a batch up to this size (six tiles of the triangle and two of scratch, 35 KB) are launched apart, so that
// they do not each hold the shared memory of the largest.
constexpr int kQeqDirectSmall = 96;

// Clusters of 8 blocks: 19 tile rows, of which a block has at most 33 tiles, besides 18 of a panel and one more.
constexpr int kQeqDirectBlocks = 8;
constexpr int kQeqDirectCluster = 608;

// Whether a block may have that much shared memory on this device (a context without it uses CG).
bool xr_qeq_direct_ready();
// One block for each of the `count` systems of `list` (device), of at most `largest` atoms. A system it
// cannot solve is left in w.qretry: [0] their number, [4 ..] the systems (adjoint: [2], [4 + S ..]).
int xr_launch_qeq_direct(const XrWork& w, const XrFF& ff, cudaStream_t st, const int* list, int count, int largest, bool adjoint);
// The same by clusters of kQeqDirectBlocks blocks; the largest system it takes on this device (0: none).
int xr_qeq_direct_cluster_max();
int xr_launch_qeq_direct_cluster(const XrWork& w, const XrFF& ff, cudaStream_t st, const int* list, int count, int largest,
                                 bool adjoint);
// The CG solver on what was left there, at most `count` systems, one block each.
int xr_launch_qeq_retry(const XrWork& w, const XrFF& ff, cudaStream_t st, int count, bool adjoint);
