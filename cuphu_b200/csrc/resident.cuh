/*
 * resident.cuh -- host interface of the on-chip Laplace solver: resident.cu
 * (mixed precision), resident_fp64.cu, and the plan (resident_plan.cu).
 */
#pragma once

#include "kernels.cuh"

#include <vector>

namespace cuphu {

constexpr int kResItemsMixed = 14;  /* work items a block can hold */
constexpr int kResItems64 = 8;
constexpr int kResMaxG = 7;         /* largest group: 2^7 blocks   */
constexpr int kResMembers = 1 << kResMaxG;

struct ResTile { int tile, g, nact, phys0; };   /* a scheduled tile: group of 2^g members,
                                                   blocks in use, its members' blocks */
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
size_t resident_mail_bytes(int nblk);
int launch_resident_mixed(const ResidentArgs &A, const TileDesc *tiles, const SolverPlanes &P,
                          SolverCtl *ctl, const SolveParams &sp, cudaStream_t s);
int launch_resident_fp64(const ResidentArgs &A, const TileDesc *tiles, const SolverPlanes &P,
                         SolverCtl *ctl, const SolveParams &sp, cudaStream_t s);

}  // namespace cuphu
