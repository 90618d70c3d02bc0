/*
 * resident.cuh -- host interface of the on-chip Laplace solver: resident.cu
 * (mixed precision), resident_fp64.cu, and the plan (resident_plan.cu).
 */
#pragma once

#include "kernels.cuh"

#include <vector>

namespace cuphu {

constexpr int kResItemsMixed = 16;  /* work items a block can hold */
constexpr int kResItems64 = 8;
constexpr int kResMaxBlocks = 160;  /* members of a group at most */
constexpr int kResMaxB = 4;         /* mixed: widest region, in items */
constexpr int kResMaxG = 7;         /* FP64: largest group, 2^7 members */
constexpr int kResMembers = 1 << kResMaxG;

/* A scheduled tile: its members (nmem entries of phys from phys0, nact of them
 * with items) and how they split it: FP64 by slots of the reduction tree
 * (2^g members), mixed precision by regions of a x b items, rcols of them per
 * row of regions. */
struct ResTile { int tile, nmem, nact, phys0, g, a, b, rcols; };
struct ResWork { int sched, member; };          /* one block's part of a scheduled tile */

/* the tiles run on the chip, in processing order, and the blocks that run
 * them; the remaining tiles go to k_solve */
struct ResidentPlan {
    std::vector<ResTile> sched;
    std::vector<unsigned short> phys;   /* block of each member (0xffff: no items) */
    std::vector<int> blk_off;           /* per block: range of work */
    std::vector<ResWork> work;
    std::vector<int> streamed;
    int nblk = 0;
};

struct ResidentArgs {                   /* the plan on the device, and scratch */
    const ResTile *sched = nullptr;
    const unsigned short *phys = nullptr;
    const int *blk_off = nullptr;
    const ResWork *work = nullptr;
    unsigned long long *rim = nullptr;
    ulonglong2 *mail = nullptr;
    unsigned *bars = nullptr;           /* one per scheduled tile, zero at launch */
    int nblk = 0;
};

void plan_resident(const std::vector<TileDesc> &tiles, int nblk, bool fp64, ResidentPlan &R);
size_t resident_rim_bytes(int nblk, bool fp64);
size_t resident_mail_bytes(int nblk, bool fp64);
int launch_resident_mixed(const ResidentArgs &A, const TileDesc *tiles, const SolverPlanes &P,
                          SolverCtl *ctl, const SolveParams &sp, cudaStream_t s);
int launch_resident_fp64(const ResidentArgs &A, const TileDesc *tiles, const SolverPlanes &P,
                         SolverCtl *ctl, const SolveParams &sp, cudaStream_t s);

}  // namespace cuphu
